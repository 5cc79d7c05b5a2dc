// Integrator drivers.
//
// Adaptive varRCWA (RedhefferIntegrator::compute + recursive_solve,
// src/core/RedhefferIntegrator.cpp:174-314, trisecting branch): every node
// [a,b] of the segmentation tree uses the eigen-basis of its own midpoint
// sample as reference, and its accept test depends on that node alone.  The
// tree is therefore explored level by level for all cells of a batch at
// once: each level evaluates every open node (one batched launch per GEMM /
// inverse / elementwise stage), the host reads back one error per node, and
// rejected nodes are replaced by their three children (two new eigen
// samples; the middle third keeps the parent's reference, as the reference
// does).  Accepted leaves are projected onto their in-order predecessor's
// basis and combined by a pairwise (tree-shaped) Redheffer star-product
// reduction, then the right end is projected onto the z1 basis.
#include "engine.h"

#include <algorithm>
#include <cmath>
#include <list>
#include <cstdlib>
#include <map>
#include <tuple>

namespace vrc {

namespace {
struct SampleB {
  int cell;
  double z;
  bool homog;
  cplx eps_h;
  cplx *P, *Q;
  int refc;
};
struct RefB {
  int sample;
  cplx *W, *V, *Winv, *Vinv, *gam;
  int refc;
};
struct NodeB {
  int cell;
  double a, b;
  int ref, sa, sm, sb, depth;
  cplx *tdd, *tuu, *rud, *rdu;
  double err;
  bool leaf;
};

struct Book {
  Engine& E;
  int n;
  const std::vector<CellSpec>& cells;
  std::vector<Engine::CellDev*>& cds;
  std::vector<SampleB> S;
  std::vector<RefB> R;
  std::vector<int> pend_samples, pend_refs;
  std::vector<int> cell_status;
  std::vector<CellResult>* out;
  // cells come four at a time, the parity classes of one mirror-symmetric
  // cell: n is the folded order, a sample is assembled once for all four
  bool folded = false;
  // of every such cell: whether a section turned out without the mirror planes.
  // Apart from the status, which later stages write; nothing takes it back.
  std::vector<char> asym;

  Book(Engine& e, int n_, const std::vector<CellSpec>& c, std::vector<Engine::CellDev*>& cd)
      : E(e), n(n_), cells(c), cds(cd) {}

  bool asymmetric(int cell) const { return folded && asym[cell / 4]; }
  int sample(int cell, double z, bool homog = false, cplx eps_h = mk(1, 0)) {
    S.push_back({cell, z, homog, eps_h, E.mat(n), E.mat(n), 0});
    pend_samples.push_back((int)S.size() - 1);
    return (int)S.size() - 1;
  }
  int ref(int s) {
    R.push_back({s, E.mat(n), E.mat(n), E.mat(n), E.mat(n), E.vec(n), 0});
    S[s].refc++;  // the eigen step reads P,Q of its sample
    pend_refs.push_back((int)R.size() - 1);
    return (int)R.size() - 1;
  }
  void release_sample(int s) {
    if (--S[s].refc == 0) {
      E.free_mat(S[s].P, n);
      E.free_mat(S[s].Q, n);
      S[s].P = S[s].Q = nullptr;
    }
  }
  void release_ref(int r) {
    if (--R[r].refc == 0) {
      E.free_mat(R[r].W, n);
      E.free_mat(R[r].V, n);
      E.free_mat(R[r].Winv, n);
      E.free_mat(R[r].Vinv, n);
      E.free_vec(R[r].gam, n);
      R[r].W = R[r].V = R[r].Winv = R[r].Vinv = R[r].gam = nullptr;
    }
  }
  // Folded samples: each distinct (structure, medium, z) is assembled at full
  // order and every class that asked for it gets its part.
  void flush_folded() {
    std::map<std::tuple<int, bool, double>, std::vector<int>> want;
    for (int s : pend_samples) {
      const SampleB& b = S[s];
      want[{b.cell / 4, b.homog, b.z}].push_back(s);
      (*out)[b.cell].n_samples++;
    }
    std::vector<std::vector<int>> groups;
    for (auto& kv : want) {  // same z, other half-space medium: a group of its own
      std::vector<std::vector<int>> part;
      for (int s : kv.second) {
        bool put = false;
        for (auto& p : part)
          if (S[p[0]].eps_h.x == S[s].eps_h.x && S[p[0]].eps_h.y == S[s].eps_h.y) {
            p.push_back(s);
            put = true;
            break;
          }
        if (!put) part.push_back({s});
      }
      for (auto& p : part) groups.push_back(std::move(p));
    }
    for (size_t g0 = 0; g0 < groups.size();) {
      const int nf = cells[S[groups[g0][0]].cell].n();  // one full order per call of a driver
      const size_t most = std::max<size_t>(1, ((size_t)512 << 20) / (32 * (size_t)nf * nf));
      const size_t g1 = std::min(groups.size(), g0 + most);
      std::vector<Engine::SampleReq> sr;
      for (size_t g = g0; g < g1; ++g) {
        const SampleB& b = S[groups[g][0]];
        sr.push_back({&cells[b.cell], cds[b.cell], b.z, b.homog, b.eps_h, E.mat(nf), E.mat(nf), nullptr, !b.homog});
      }
      std::vector<int> st;
      E.assemble(sr, &st);
      std::map<std::pair<int, int>, std::vector<FoldDesc>> fd;  // by harmonic counts
      for (size_t g = g0; g < g1; ++g)
        for (int s : groups[g]) {
          const SampleB& b = S[s];
          const CellSpec& c = cells[b.cell];
          fd[{c.nx, c.ny}].push_back({sr[g - g0].P, sr[g - g0].Q, b.P, b.Q, c.k0() * c.k0(), b.cell % 4});
          if (st[g - g0] == ST_ASYMMETRIC || (!b.homog && c.kind != GEOM_PILLAR && !c.mirrored(b.z)))
            asym[b.cell / 4] = 1;
          else if (st[g - g0])
            cell_status[b.cell] = st[g - g0];
        }
      for (auto& kv : fd) {
        const FoldDesc* d = E.upload(kv.second);
        Engine::Prof pr(E, "assembly", 0.0, 160.0 * n * (double)n * kv.second.size());
        fold_batched(d, (int)kv.second.size(), kv.first.first, kv.first.second, E.stream());
      }
      for (auto& r : sr) {
        E.free_mat(r.P, nf);
        E.free_mat(r.Q, nf);
      }
      g0 = g1;
    }
  }
  // Assemble all pending samples and decompose all pending references.
  void flush() {
    std::vector<int> st;
    if (folded) {
      flush_folded();
    } else {
      std::vector<Engine::SampleReq> sr;
      for (int s : pend_samples) {
        const SampleB& b = S[s];
        sr.push_back({&cells[b.cell], cds[b.cell], b.z, b.homog, b.eps_h, b.P, b.Q});
        (*out)[b.cell].n_samples++;
      }
      E.assemble(sr, &st);
      for (size_t i = 0; i < st.size(); ++i)
        if (st[i]) cell_status[S[pend_samples[i]].cell] = st[i];
    }
    std::vector<Engine::EigReq> er;
    for (int r : pend_refs) {
      const RefB& b = R[r];
      er.push_back({S[b.sample].P, S[b.sample].Q, b.W, b.V, b.Winv, b.Vinv, b.gam});
      (*out)[S[b.sample].cell].n_eig++;
    }
    st.clear();
    E.eig(er, n, &st);
    for (size_t i = 0; i < st.size(); ++i)
      if (st[i]) cell_status[S[R[pend_refs[i]].sample].cell] = st[i];
    for (int r : pend_refs) release_sample(R[r].sample);
    pend_samples.clear();
    pend_refs.clear();
  }
  int end_basis(int cell, int own_sample, bool has, cplx eps) {
    int s = own_sample;
    if (has) s = sample(cell, cells[cell].z0, true, eps);
    int r = ref(s);
    R[r].refc++;  // held by the cell until the end
    return r;
  }
  void export_basis(int r, cplx*& W, cplx*& V, cplx*& gam, cplx*& Winv) {
    W = R[r].W;
    V = R[r].V;
    gam = R[r].gam;
    Winv = R[r].Winv;
    E.free_mat(R[r].Vinv, n);
    R[r].W = R[r].V = R[r].gam = R[r].Winv = R[r].Vinv = nullptr;
  }
};

void start_results(const std::vector<CellSpec>& cells, std::vector<CellResult>& out) {
  out.assign(cells.size(), CellResult());
  for (size_t c = 0; c < cells.size(); ++c) out[c].n = cells[c].n();
}

// Order of the problems solved for cells of order n.
int solved_order(int n, int folded) { return folded ? (n / 2 + 1) / 2 : n; }

// Cells whose S-matrix is wanted.  FOLD_EXCITED: the classes that a normally
// incident plane wave excites, (even, even) by x polarisation and (odd, odd) by
// y polarisation.
bool excited(int c, int folded) { return folded != Engine::FOLD_EXCITED || c % 4 == 0 || c % 4 == 3; }

// The four classes of a cell share its CellDev.
std::vector<Engine::CellDev*> prepare_cells(Engine& E, const std::vector<CellSpec>& cells, int folded) {
  std::vector<Engine::CellDev*> cds;
  for (size_t c = 0; c < cells.size(); ++c)
    cds.push_back(folded && c % 4 ? cds.back() : E.prepare_cell(cells[c]));
  return cds;
}
void release_cells(Engine& E, const std::vector<Engine::CellDev*>& cds, int folded) {
  for (size_t c = 0; c < cds.size(); ++c)
    if (!folded || c % 4 == 0) E.release_cell(cds[c]);
}

void validate(const CellSpec& c) {
  if (c.kind == GEOM_SAMPLER) {
    // only n = 2 nx ny matters to the integrators (a LayerSampler exposes nDim)
    if (c.nx < 1 || c.ny < 1 || c.n() > 1024) throw StatusError(ST_EINVAL, "sampler cell: need 2 <= n <= 1024");
    if (!c.host_sample && !c.dev_sample) throw StatusError(ST_EINVAL, "sampler cell without a sampler callback");
    if (!(c.lambda > 0.0)) throw StatusError(ST_EINVAL, "wavelength must be positive");
    if ((c.has_end0 || c.has_end1) && ((c.nx % 2) == 0 || (c.ny % 2) == 0 || c.nx > 64 || c.ny > 64))
      throw StatusError(ST_EINVAL, "half-space ends need the odd harmonic counts nx, ny of the sampler");
    return;
  }
  if (c.nx < 1 || c.ny < 1 || (c.nx % 2) == 0 || (c.ny % 2) == 0)
    throw StatusError(ST_EINVAL, "harmonic counts must be odd and positive");
  if (c.nx > 64 || c.ny > 64 || c.n() > 1024)
    throw StatusError(ST_EINVAL, "truncation too large (nx, ny <= 64 and n <= 1024)");
  if (!(c.lambda > 0.0)) throw StatusError(ST_EINVAL, "wavelength must be positive");
  if (c.kind == GEOM_PILLAR) {
    if (c.npx < 1 || c.npy < 1) throw StatusError(ST_EINVAL, "pillar raster must be non-empty");
  } else if (c.kind == GEOM_PLANAR) {
    if (c.polys.empty()) throw StatusError(ST_EINVAL, "planar cell needs polygons");
    for (const auto& p : c.polys)
      if (p.size() < 6 || p.size() % 2) throw StatusError(ST_EINVAL, "planar polygons need >= 3 points");
    if (!(c.thickness > 0.0)) throw StatusError(ST_EINVAL, "planar device thickness must be positive");
    for (int q = 0; q < 4; ++q)
      if (!(c.pml_w[q] > 0.0) || !(c.space[q] >= 0.0)) throw StatusError(ST_EINVAL, "planar PML / spaces invalid");
  } else {
    if (c.x.size() < 2 || c.y.size() < 2) throw StatusError(ST_EINVAL, "grid needs at least 2 coordinates per axis");
    if (c.eps.size() != (c.x.size() - 1) * (c.y.size() - 1))
      throw StatusError(ST_EINVAL, "eps table does not match the coordinates");
    if (c.pml && (c.x.size() < 4 || c.y.size() < 4))
      throw StatusError(ST_EINVAL, "PML needs at least 4 coordinates per axis");
    for (const auto& r : c.xrules)
      if (r.index < 0 || r.index >= (int)c.x.size() || r.zs.size() != r.vals.size() || r.zs.empty())
        throw StatusError(ST_EINVAL, "invalid x rule");
    for (const auto& r : c.yrules)
      if (r.index < 0 || r.index >= (int)c.y.size() || r.zs.size() != r.vals.size() || r.zs.empty())
        throw StatusError(ST_EINVAL, "invalid y rule");
  }
}
}  // namespace

void Engine::release_result(CellResult& r) {
  const int n = r.n;
  free_mat(r.Tdd, n); free_mat(r.Tuu, n); free_mat(r.Rud, n); free_mat(r.Rdu, n);
  free_mat(r.W0, n); free_mat(r.V0, n); free_vec(r.gam0, n); free_mat(r.W0inv, n);
  free_mat(r.W1, n); free_mat(r.V1, n); free_vec(r.gam1, n); free_mat(r.W1inv, n);
  r.Tdd = r.Tuu = r.Rud = r.Rdu = r.W0 = r.V0 = r.gam0 = r.W0inv = r.W1 = r.V1 = r.gam1 = r.W1inv = nullptr;
}

// ---------------------------------------------------------------------------
// Adaptive varRCWA
// ---------------------------------------------------------------------------
void Engine::redheffer(const std::vector<CellSpec>& cells, const RedhefferOpts& o, std::vector<CellResult>& out) {
  const int folded = o.folded;
  for (const auto& c : cells) validate(c);
  start_results(cells, out);
  std::map<int, std::vector<int>> by_n;
  for (size_t c = 0; c < cells.size(); ++c) by_n[cells[c].n()].push_back((int)c);
  std::vector<std::pair<int, std::vector<int>>> classes(by_n.begin(), by_n.end());
  if (!classes.empty())
    std::rotate(classes.begin(), classes.begin() + (size_t)std::max(0, o.rotate) % classes.size(), classes.end());
  for (auto& kv : classes) {
    const int n = solved_order(kv.first, folded);
    const std::vector<int>& ids = kv.second;
    std::vector<CellSpec> sub;
    for (int c : ids) sub.push_back(cells[c]);
    std::vector<CellDev*> cds = prepare_cells(*this, sub, folded);
    std::vector<CellResult> res(sub.size());
    for (size_t c = 0; c < sub.size(); ++c) res[c].n = n;
    Book bk(*this, n, sub, cds);
    bk.out = &res;
    bk.folded = folded != 0;
    bk.asym.assign(sub.size() / 4 + 1, 0);
    bk.cell_status.assign(sub.size(), ST_OK);
    const int C = (int)sub.size();
    std::vector<NodeB> N;
    std::vector<std::list<int>> order(C);
    std::vector<int> e0(C), e1(C);
    std::vector<int> active;
    for (int c = 0; c < C; ++c) {
      const CellSpec& s = sub[c];
      const double z0 = s.z0, z1 = s.z1;
      const int s0 = bk.sample(c, z0), s1 = bk.sample(c, z1);
      e0[c] = bk.end_basis(c, s0, s.has_end0, s.eps_end0);
      e1[c] = bk.end_basis(c, s1, s.has_end1, s.eps_end1);
      if (o.cuts && !(*o.cuts)[ids[c]].empty()) {
        // explicit segments: each with its own midpoint reference
        const std::vector<double>& cut = (*o.cuts)[ids[c]];
        int sa = s0;
        for (size_t k = 0; k + 1 < cut.size(); ++k) {
          double a = cut[k], b = cut[k + 1];
          int sm = bk.sample(c, 0.5 * (a + b));
          int sb = (k + 2 == cut.size()) ? s1 : bk.sample(c, b);
          int r = bk.ref(sm);
          NodeB nd{c, a, b, r, sa, sm, sb, 0, nullptr, nullptr, nullptr, nullptr, 0.0, false};
          bk.R[r].refc++;
          bk.S[sa].refc++;
          bk.S[sm].refc++;
          bk.S[sb].refc++;
          N.push_back(nd);
          order[c].push_back((int)N.size() - 1);
          active.push_back((int)N.size() - 1);
          sa = sb;
        }
      } else {
        const double zm = 0.5 * (z0 + z1);
        const int sm = bk.sample(c, zm);
        const int r = bk.ref(sm);
        NodeB nd{c, z0, z1, r, s0, sm, s1, 0, nullptr, nullptr, nullptr, nullptr, 0.0, false};
        bk.R[r].refc++;
        bk.S[s0].refc++;
        bk.S[sm].refc++;
        bk.S[s1].refc++;
        N.push_back(nd);
        order[c].push_back(0 + (int)N.size() - 1);
        active.push_back((int)N.size() - 1);
      }
    }
    bk.flush();
    // An asymmetric cell's classes are not a problem worth solving: its tree ends
    // here, and the caller takes it the general way.
    auto drop_asymmetric = [&] {
      if (!folded) return;
      for (int id : active) {
        const NodeB& nd = N[id];
        if (!bk.asymmetric(nd.cell)) continue;
        bk.release_sample(nd.sa);
        bk.release_sample(nd.sm);
        bk.release_sample(nd.sb);
      }
      active.erase(std::remove_if(active.begin(), active.end(), [&](int id) { return bk.asymmetric(N[id].cell); }),
                   active.end());
      for (int c = 0; c < C; ++c) {
        if (!bk.asymmetric(c)) continue;
        for (int id : order[c]) {
          free_mat(N[id].tdd, n); free_mat(N[id].tuu, n); free_mat(N[id].rud, n); free_mat(N[id].rdu, n);
          bk.release_ref(N[id].ref);
        }
        order[c].clear();
      }
    };
    drop_asymmetric();
    const bool replay = (o.cuts != nullptr);
    while (!active.empty()) {
      // Evaluate every open node of this level.
      double* derr = (double*)bytes(active.size() * sizeof(double));
      VRC_CUDA_CHECK(cudaMemsetAsync(derr, 0, active.size() * sizeof(double), stream_));
      std::vector<SegReq> sr;
      for (size_t i = 0; i < active.size(); ++i) {
        NodeB& nd = N[active[i]];
        nd.tdd = mat(n); nd.tuu = mat(n); nd.rud = mat(n); nd.rdu = mat(n);
        const RefB& r = bk.R[nd.ref];
        const SampleB& sm = bk.S[nd.sm];
        sr.push_back({sm.P, sm.Q, r.W, r.V, r.Winv, r.Vinv, r.gam, bk.S[nd.sa].P, bk.S[nd.sa].Q, bk.S[nd.sb].P,
                      bk.S[nd.sb].Q, nd.a, nd.b, sub[nd.cell].k0(), nd.tdd, nd.tuu, nd.rud, nd.rdu, derr + i});
      }
      segments(sr, n);
      std::vector<double> herr(active.size());
      VRC_CUDA_CHECK(cudaMemcpyAsync(herr.data(), derr, herr.size() * sizeof(double), cudaMemcpyDeviceToHost, stream_));
      sync();
      free_bytes(derr, active.size() * sizeof(double));
      if (folded) {  // a node's error is the largest of its four classes
        std::map<std::pair<int, double>, double> worst;
        for (size_t i = 0; i < active.size(); ++i) {
          const NodeB& nd = N[active[i]];
          auto it = worst.emplace(std::make_pair(nd.cell / 4, nd.a), herr[i]).first;
          if (!(herr[i] <= it->second) && !std::isnan(it->second)) it->second = herr[i];
        }
        for (size_t i = 0; i < active.size(); ++i) herr[i] = worst[{N[active[i]].cell / 4, N[active[i]].a}];
      }
      std::vector<int> next;
      for (size_t i = 0; i < active.size(); ++i) {
        const int id = active[i];
        NodeB nd = N[id];
        nd.err = herr[i];
        const bool accept = replay || nd.err <= o.pe || nd.depth >= o.max_depth;
        res[nd.cell].nodes.push_back({nd.a, nd.b, nd.err, accept ? 1 : 0});
        res[nd.cell].n_nodes++;
        if (!std::isfinite(nd.err)) bk.cell_status[nd.cell] = ST_ENONFINITE;
        if (accept) {
          nd.leaf = true;
          if (nd.depth >= o.max_depth && nd.err > o.pe && !replay) bk.cell_status[nd.cell] = ST_EDEPTH;
          res[nd.cell].N++;
          N[id] = nd;
          bk.release_sample(nd.sa);
          bk.release_sample(nd.sm);
          bk.release_sample(nd.sb);
          continue;
        }
        free_mat(nd.tdd, n); free_mat(nd.tuu, n); free_mat(nd.rud, n); free_mat(nd.rdu, n);
        nd.tdd = nd.tuu = nd.rud = nd.rdu = nullptr;
        const int c = nd.cell;
        const double a = nd.a, b = nd.b;
        const double zm0 = 2. / 3. * a + 1. / 3. * b;
        const double zm1 = 1. / 3. * a + 2. / 3. * b;
        const int st = bk.sample(c, 0.5 * (a + zm0));
        const int sk = bk.sample(c, zm0);
        const int st2 = bk.sample(c, zm1);
        const int sk2 = bk.sample(c, 0.5 * (zm1 + b));
        const int rl = bk.ref(st), rr = bk.ref(sk2);
        NodeB L{c, a, zm0, rl, nd.sa, st, sk, nd.depth + 1, nullptr, nullptr, nullptr, nullptr, 0.0, false};
        NodeB M{c, zm0, zm1, nd.ref, sk, nd.sm, st2, nd.depth + 1, nullptr, nullptr, nullptr, nullptr, 0.0, false};
        NodeB Rn{c, zm1, b, rr, st2, sk2, nd.sb, nd.depth + 1, nullptr, nullptr, nullptr, nullptr, 0.0, false};
        for (const NodeB* ch : {&L, &M, &Rn}) {
          bk.R[ch->ref].refc++;
          bk.S[ch->sa].refc++;
          bk.S[ch->sm].refc++;
          bk.S[ch->sb].refc++;
        }
        N.push_back(L);
        const int il = (int)N.size() - 1;
        N.push_back(M);
        const int im = (int)N.size() - 1;
        N.push_back(Rn);
        const int ir = (int)N.size() - 1;
        auto it = std::find(order[c].begin(), order[c].end(), id);
        it = order[c].erase(it);
        order[c].insert(it, {il, im, ir});
        next.push_back(il);
        next.push_back(im);
        next.push_back(ir);
        bk.release_ref(nd.ref);
        bk.release_sample(nd.sa);
        bk.release_sample(nd.sm);
        bk.release_sample(nd.sb);
        N[id] = nd;
      }
      bk.flush();
      active.swap(next);
      drop_asymmetric();
    }
    // Left-end projections of all leaves onto their predecessors' bases.
    std::vector<ProjReq> pr;
    std::vector<int> pr_cell;
    for (int c = 0; c < C; ++c) {
      if (!excited(c, folded)) {  // only its errors were needed
        for (int id : order[c]) {
          free_mat(N[id].tdd, n); free_mat(N[id].tuu, n); free_mat(N[id].rud, n); free_mat(N[id].rdu, n);
          bk.release_ref(N[id].ref);
        }
        order[c].clear();
        continue;
      }
      int prev = e0[c];
      for (int id : order[c]) {
        const NodeB& nd = N[id];
        const RefB& r = bk.R[nd.ref];
        pr.push_back({r.Winv, r.Vinv, bk.R[prev].W, bk.R[prev].V, nd.tdd, nd.tuu, nd.rud, nd.rdu});
        pr_cell.push_back(c);
        prev = nd.ref;
      }
    }
    std::vector<int> pst;
    project_left(pr, n, &pst);
    for (size_t i = 0; i < pst.size(); ++i)
      if (pst[i]) bk.cell_status[pr_cell[i]] = pst[i];
    std::vector<std::vector<SBlocks>> lists(C);
    std::vector<int> last(C);
    for (int c = 0; c < C; ++c) {
      if (order[c].empty()) continue;
      for (int id : order[c]) lists[c].push_back({N[id].tdd, N[id].tuu, N[id].rud, N[id].rdu});
      last[c] = N[order[c].back()].ref;
      for (int id : order[c])
        if (N[id].ref != last[c]) bk.release_ref(N[id].ref);
    }
    star_reduce(lists, n, &bk.cell_status);
    std::vector<ProjRReq> rr;
    std::vector<int> rr_cell;
    for (int c = 0; c < C; ++c) {
      if (lists[c].empty()) continue;
      rr_cell.push_back(c);
      const SBlocks& s = lists[c][0];
      rr.push_back({bk.R[last[c]].Winv, bk.R[last[c]].Vinv, bk.R[e1[c]].W, bk.R[e1[c]].V, s.tdd, s.tuu, s.rud, s.rdu});
    }
    std::vector<int> rst;
    project_right(rr, n, &rst);
    sync();
    for (size_t i = 0; i < rst.size(); ++i)
      if (rst[i]) bk.cell_status[rr_cell[i]] = rst[i];
    for (int c = 0; c < C; ++c) {
      // release the remaining holds of the last leaf's reference
      for (int id : order[c])
        if (N[id].ref == last[c]) bk.release_ref(last[c]);
      CellResult& r = res[c];
      if (!lists[c].empty()) {
        r.Tdd = lists[c][0].tdd;
        r.Tuu = lists[c][0].tuu;
        r.Rud = lists[c][0].rud;
        r.Rdu = lists[c][0].rdu;
      }
      bk.export_basis(e0[c], r.W0, r.V0, r.gam0, r.W0inv);
      bk.export_basis(e1[c], r.W1, r.V1, r.gam1, r.W1inv);
      r.status = bk.asymmetric(c) ? (int)ST_ASYMMETRIC : bk.cell_status[c];
    }
    // samples still referenced by end bases
    for (size_t s = 0; s < bk.S.size(); ++s)
      if (bk.S[s].P) {
        free_mat(bk.S[s].P, n);
        free_mat(bk.S[s].Q, n);
      }
    release_cells(*this, cds, folded);
    for (size_t c = 0; c < ids.size(); ++c) out[ids[c]] = res[c];
  }
}

// ---------------------------------------------------------------------------
// Plain RCWA: N midpoint slices (RCWAIntegrator::compute,
// src/core/RCWAIntegrator.cpp:20-87).
// ---------------------------------------------------------------------------
void Engine::rcwa(const std::vector<CellSpec>& cells, int Nsl, std::vector<CellResult>& out, int folded) {
  if (Nsl < 1) throw StatusError(ST_EINVAL, "N must be >= 1");
  for (const auto& c : cells) validate(c);
  start_results(cells, out);
  std::map<int, std::vector<int>> by_n;
  for (size_t c = 0; c < cells.size(); ++c) by_n[cells[c].n()].push_back((int)c);
  for (auto& kv : by_n) {
    const int n = solved_order(kv.first, folded);
    const std::vector<int>& ids = kv.second;
    std::vector<CellSpec> sub;
    for (int c : ids) sub.push_back(cells[c]);
    std::vector<CellDev*> cds = prepare_cells(*this, sub, folded);
    std::vector<CellResult> res(sub.size());
    for (auto& r : res) r.n = n;
    Book bk(*this, n, sub, cds);
    bk.out = &res;
    bk.folded = folded != 0;
    bk.asym.assign(sub.size() / 4 + 1, 0);
    const int C = (int)sub.size();
    bk.cell_status.assign(C, ST_OK);
    std::vector<int> e0(C), e1(C);
    std::vector<std::vector<int>> slices(C);
    for (int c = 0; c < C; ++c) {
      if (!excited(c, folded)) continue;
      const CellSpec& s = sub[c];
      const int s1 = bk.sample(c, s.z1);
      e1[c] = bk.end_basis(c, s1, s.has_end1, s.eps_end1);
      const double dz = (s.z1 - s.z0) / (double)Nsl;
      for (int i = 0; i < Nsl; ++i) {
        int si = bk.sample(c, s.z0 + (i + 0.5) * dz);
        bk.S[si].refc++;
        slices[c].push_back(si);
      }
      const int s0 = bk.sample(c, s.z0);
      e0[c] = bk.end_basis(c, s0, s.has_end0, s.eps_end0);
    }
    bk.flush();
    std::vector<SlabReq> sl;
    std::vector<std::vector<SBlocks>> lists(C);
    std::vector<int> sl_cell;
    for (int c = 0; c < C; ++c) {
      if (!excited(c, folded) || bk.asymmetric(c)) continue;
      const CellSpec& s = sub[c];
      const double dz = (s.z1 - s.z0) / (double)Nsl;
      for (int si : slices[c]) {
        SBlocks b{mat(n), mat(n), mat(n), mat(n)};
        sl.push_back({bk.S[si].P, bk.S[si].Q, bk.R[e1[c]].W, bk.R[e1[c]].V, s.k0(), dz, b.tuu, b.rud});
        sl_cell.push_back(c);
        lists[c].push_back(b);
      }
      res[c].n_eig += Nsl;
      res[c].N = Nsl;
    }
    std::vector<int> sst;
    rcwa_slabs(sl, n, &sst);
    for (size_t i = 0; i < sst.size(); ++i)
      if (sst[i]) bk.cell_status[sl_cell[i]] = sst[i];
    // symmetric slab: tdd = tuu, rdu = rud (RCWAScatterMatrix.h:44-47)
    std::vector<cplx*> src, dst;
    for (auto& L : lists)
      for (auto& b : L) {
        src.push_back(b.tuu); dst.push_back(b.tdd);
        src.push_back(b.rud); dst.push_back(b.rdu);
      }
    copy(src, dst, n);
    for (int c = 0; c < C; ++c)
      for (int si : slices[c]) bk.release_sample(si);
    star_reduce(lists, n, &bk.cell_status);
    std::vector<ProjLEReq> pl;
    std::vector<int> pl_cell;
    for (int c = 0; c < C; ++c) {
      if (lists[c].empty()) continue;
      pl_cell.push_back(c);
      const SBlocks& s = lists[c][0];
      pl.push_back({bk.R[e1[c]].Winv, bk.R[e1[c]].Vinv, bk.R[e0[c]].W, bk.R[e0[c]].V, s.tdd, s.tuu, s.rud, s.rdu});
    }
    std::vector<int> pst;
    project_left_end(pl, n, &pst);
    sync();
    for (size_t i = 0; i < pst.size(); ++i)
      if (pst[i]) bk.cell_status[pl_cell[i]] = pst[i];
    for (int c = 0; c < C; ++c) {
      CellResult& r = res[c];
      if (!excited(c, folded)) continue;
      if (!lists[c].empty()) {
        r.Tdd = lists[c][0].tdd; r.Tuu = lists[c][0].tuu; r.Rud = lists[c][0].rud; r.Rdu = lists[c][0].rdu;
      }
      bk.export_basis(e0[c], r.W0, r.V0, r.gam0, r.W0inv);
      bk.export_basis(e1[c], r.W1, r.V1, r.gam1, r.W1inv);
      r.status = bk.asymmetric(c) ? (int)ST_ASYMMETRIC : bk.cell_status[c];
    }
    for (size_t s = 0; s < bk.S.size(); ++s)
      if (bk.S[s].P) { free_mat(bk.S[s].P, n); free_mat(bk.S[s].Q, n); }
    release_cells(*this, cds, folded);
    for (size_t c = 0; c < ids.size(); ++c) out[ids[c]] = res[c];
  }
}

// ---------------------------------------------------------------------------
// Differential method (DifferentialIntegrator::compute,
// src/core/DifferentialIntegrator.cpp:21-134).
// ---------------------------------------------------------------------------
void Engine::differential(const std::vector<CellSpec>& cells, int Nsl, std::vector<CellResult>& out, int folded) {
  if (Nsl < 1) throw StatusError(ST_EINVAL, "N must be >= 1");
  for (const auto& c : cells) validate(c);
  start_results(cells, out);
  std::map<int, std::vector<int>> by_n;
  for (size_t c = 0; c < cells.size(); ++c) by_n[cells[c].n()].push_back((int)c);
  for (auto& kv : by_n) {
    const int n = solved_order(kv.first, folded);
    const std::vector<int>& ids = kv.second;
    std::vector<CellSpec> sub;
    for (int c : ids) sub.push_back(cells[c]);
    std::vector<CellDev*> cds = prepare_cells(*this, sub, folded);
    std::vector<CellResult> res(sub.size());
    for (auto& r : res) r.n = n;
    Book bk(*this, n, sub, cds);
    bk.out = &res;
    bk.folded = folded != 0;
    bk.asym.assign(sub.size() / 4 + 1, 0);
    const int C = (int)sub.size();
    bk.cell_status.assign(C, ST_OK);
    std::vector<int> e0(C), e1(C);
    std::vector<std::vector<int>> pts(C);  // samples at z0, zm_0, zr_0, zm_1, zr_1, ...
    for (int c = 0; c < C; ++c) {
      if (!excited(c, folded)) continue;
      const CellSpec& s = sub[c];
      const int s1 = bk.sample(c, s.z1);
      e1[c] = bk.end_basis(c, s1, s.has_end1, s.eps_end1);
      const double dz = (s.z1 - s.z0) / (double)Nsl;
      int p0 = bk.sample(c, s.z0);
      bk.S[p0].refc++;
      pts[c].push_back(p0);
      for (int i = 0; i < Nsl; ++i) {
        const double zl = s.z0 + i * dz, zr = s.z0 + (i + 1) * dz, zm = 0.5 * (zl + zr);
        int pm = bk.sample(c, zm), pr = bk.sample(c, zr);
        bk.S[pm].refc++;
        bk.S[pr].refc++;
        pts[c].push_back(pm);
        pts[c].push_back(pr);
      }
      const int s0 = bk.sample(c, s.z0);
      e0[c] = bk.end_basis(c, s0, s.has_end0, s.eps_end0);
      res[c].N = Nsl;
    }
    bk.flush();
    std::vector<DiffReq> dr;
    std::vector<std::vector<SBlocks>> lists(C);
    std::vector<int> dr_cell;
    for (int c = 0; c < C; ++c) {
      if (!excited(c, folded) || bk.asymmetric(c)) continue;
      const CellSpec& s = sub[c];
      const double dz = (s.z1 - s.z0) / (double)Nsl;
      const RefB& b1 = bk.R[e1[c]];
      for (int i = 0; i < Nsl; ++i) {
        const SampleB &A0 = bk.S[pts[c][2 * i]], &A1 = bk.S[pts[c][2 * i + 1]], &A2 = bk.S[pts[c][2 * i + 2]];
        SBlocks b{mat(n), mat(n), mat(n), mat(n)};
        dr.push_back({A0.P, A0.Q, A1.P, A1.Q, A2.P, A2.Q, b1.W, b1.V, b1.Winv, b1.Vinv, s.k0(), dz, b.tdd, b.tuu, b.rud,
                      b.rdu});
        dr_cell.push_back(c);
        lists[c].push_back(b);
      }
    }
    std::vector<int> dst;
    diff_slices(dr, n, &dst);
    for (size_t i = 0; i < dst.size(); ++i)
      if (dst[i]) bk.cell_status[dr_cell[i]] = dst[i];
    for (int c = 0; c < C; ++c)
      for (int p : pts[c]) bk.release_sample(p);
    star_reduce(lists, n, &bk.cell_status);
    std::vector<ProjLEReq> pl;
    std::vector<int> pl_cell;
    for (int c = 0; c < C; ++c) {
      if (lists[c].empty()) continue;
      pl_cell.push_back(c);
      const SBlocks& s = lists[c][0];
      pl.push_back({bk.R[e1[c]].Winv, bk.R[e1[c]].Vinv, bk.R[e0[c]].W, bk.R[e0[c]].V, s.tdd, s.tuu, s.rud, s.rdu});
    }
    std::vector<int> pst;
    project_left_end(pl, n, &pst);
    sync();
    for (size_t i = 0; i < pst.size(); ++i)
      if (pst[i]) bk.cell_status[pl_cell[i]] = pst[i];
    for (int c = 0; c < C; ++c) {
      CellResult& r = res[c];
      if (!excited(c, folded)) continue;
      if (!lists[c].empty()) {
        r.Tdd = lists[c][0].tdd; r.Tuu = lists[c][0].tuu; r.Rud = lists[c][0].rud; r.Rdu = lists[c][0].rdu;
      }
      bk.export_basis(e0[c], r.W0, r.V0, r.gam0, r.W0inv);
      bk.export_basis(e1[c], r.W1, r.V1, r.gam1, r.W1inv);
      r.status = bk.asymmetric(c) ? (int)ST_ASYMMETRIC : bk.cell_status[c];
    }
    for (size_t s = 0; s < bk.S.size(); ++s)
      if (bk.S[s].P) { free_mat(bk.S[s].P, n); free_mat(bk.S[s].Q, n); }
    release_cells(*this, cds, folded);
    for (size_t c = 0; c < ids.size(); ++c) out[ids[c]] = res[c];
  }
}

// ---------------------------------------------------------------------------
// Per-order powers (RCWASolver::scatterPlaneWave, src/rcwa/RCWASolver.cpp:1636-1733)
// ---------------------------------------------------------------------------
void Engine::order_powers(const std::vector<CellSpec>& cells, const std::vector<CellResult>& res, int side,
                          int flux_norm, std::vector<std::vector<double>>& Rout,
                          std::vector<std::vector<double>>& Tout, int folded) {
  const size_t C = cells.size();
  Rout.assign(C, {});
  Tout.assign(C, {});
  std::map<int, std::vector<int>> by_n;
  for (size_t c = 0; c < C; ++c) {
    if (!cells[c].has_end0 || !cells[c].has_end1)
      throw StatusError(ST_EINVAL, "order powers need homogeneous end media");
    if (cells[c].pml) throw StatusError(ST_EINVAL, "order powers need periodic boundaries");
    by_n[cells[c].n()].push_back((int)c);
  }
  for (auto& kv : by_n) {
    const int n = kv.first, m = n / 2;
    const std::vector<int>& ids = kv.second;
    const size_t B = ids.size();
    // two polarisations per cell
    std::vector<cplx*> cvec(2 * B), rc(2 * B), rf(2 * B), tc(2 * B), tf(2 * B);
    std::vector<MatVecDesc> mv1, mv2;
    std::vector<double*> Rd(2 * B), Td(2 * B);
    std::vector<double*> ab(B);
    const int ns = solved_order(n, folded);
    std::vector<cplx*> cls;  // folded: the classes' harmonics
    std::map<std::pair<int, int>, std::vector<UnfoldDesc>> ud;
    for (size_t b = 0; b < B; ++b) {
      const CellSpec& s = cells[ids[b]];
      const int nx = s.nx, ny = s.ny;
      for (int p = 0; p < 2; ++p) {
        const size_t k = 2 * b + p;
        // the class of this polarisation, and its zero order's place there
        const CellResult& r = folded ? res[4 * ids[b] + (p == 0 ? 0 : 3)] : res[ids[b]];
        const int c0 = folded ? (p == 0 ? 0 : (nx - 1) / 2 * ((ny - 1) / 2))
                              : (p == 0 ? 0 : m) + (ny * (nx - 1)) / 2 + (ny - 1) / 2;
        const cplx* Win = side == 0 ? r.W0 : r.W1;
        const cplx* Wininv = side == 0 ? r.W0inv : r.W1inv;
        const cplx* Wout = side == 0 ? r.W1 : r.W0;
        const cplx* Rm = side == 0 ? r.Rdu : r.Rud;
        const cplx* Tm = side == 0 ? r.Tuu : r.Tdd;
        // c = Win^-1 s with s the unit vector of the zero order (px or py)
        cvec[k] = const_cast<cplx*>(Wininv) + (size_t)c0 * ns;
        rc[k] = vec(n); rf[k] = vec(n); tc[k] = vec(n); tf[k] = vec(n);
        cplx *rk = rf[k], *tk = tf[k];
        if (folded) {
          cls.push_back(rk = vec(n));
          cls.push_back(tk = vec(n));
          ud[{nx, ny}].push_back({rk, rf[k], p == 0 ? 0 : 3});
          ud[{nx, ny}].push_back({tk, tf[k], p == 0 ? 0 : 3});
        }
        mv1.push_back({Rm, cvec[k], rc[k]});
        mv1.push_back({Tm, cvec[k], tc[k]});
        mv2.push_back({Win, rc[k], rk});
        mv2.push_back({Wout, tc[k], tk});
        Rd[k] = (double*)bytes(m * sizeof(double));
        Td[k] = (double*)bytes(m * sizeof(double));
      }
      ab[b] = (double*)bytes(2 * m * sizeof(double));
    }
    {
      const double work = 16.0 * ns * (double)ns * (mv1.size() + mv2.size());
      Prof pr(*this, "powers", work, work, 2 + (int)ud.size());
      matvec_batched(upload(mv1), (int)mv1.size(), ns, stream_);
      matvec_batched(upload(mv2), (int)mv2.size(), ns, stream_);
      for (auto& kv : ud)
        unfold_batched(upload(kv.second), (int)kv.second.size(), kv.first.first, kv.first.second, stream_);
    }
    std::vector<PowerDesc> pd;
    std::vector<std::vector<double>> hab(B);
    for (size_t b = 0; b < B; ++b) {
      const CellSpec& s = cells[ids[b]];
      // alpha/beta: src/core/LayerSampler.cpp:9-32
      std::vector<double> x, y;
      s.geometry(s.z0, x, y);
      const double Lx = x.back() - x.front(), Ly = y.back() - y.front();
      hab[b].resize(2 * m);
      const int Nx = (s.nx - 1) / 2, Ny = (s.ny - 1) / 2;
      for (int i = 0; i < s.nx; ++i)
        for (int j = 0; j < s.ny; ++j) {
          hab[b][s.ny * i + j] = (2 * 3.1415926535897932 / Lx) * (double)(i - Nx);
          hab[b][m + s.ny * i + j] = (2 * 3.1415926535897932 / Ly) * (double)(j - Ny);
        }
      VRC_CUDA_CHECK(cudaMemcpyAsync(ab[b], hab[b].data(), 2 * m * sizeof(double), cudaMemcpyHostToDevice, stream_));
      const cplx ein = side == 0 ? s.eps_end0 : s.eps_end1;
      const cplx eout = side == 0 ? s.eps_end1 : s.eps_end0;
      const double tn = flux_norm ? std::sqrt(ein.x) : std::sqrt(eout.x);
      for (int p = 0; p < 2; ++p) {
        const size_t k = 2 * b + p;
        pd.push_back({rf[k], tf[k], ab[b], ab[b] + m, Rd[k], Td[k], ein, eout, s.k0(), tn});
      }
    }
    {
      Prof pr(*this, "powers", 0.0, 64.0 * m * (double)pd.size());
      order_power_batched(upload(pd), (int)pd.size(), m, stream_);
    }
    for (size_t b = 0; b < B; ++b) {
      Rout[ids[b]].resize(2 * m);
      Tout[ids[b]].resize(2 * m);
      for (int p = 0; p < 2; ++p) {
        const size_t k = 2 * b + p;
        VRC_CUDA_CHECK(cudaMemcpyAsync(Rout[ids[b]].data() + p * m, Rd[k], m * sizeof(double), cudaMemcpyDeviceToHost,
                                       stream_));
        VRC_CUDA_CHECK(cudaMemcpyAsync(Tout[ids[b]].data() + p * m, Td[k], m * sizeof(double), cudaMemcpyDeviceToHost,
                                       stream_));
      }
    }
    sync();
    for (size_t k = 0; k < 2 * B; ++k) {
      free_vec(rc[k], n); free_vec(rf[k], n); free_vec(tc[k], n); free_vec(tf[k], n);
      free_bytes(Rd[k], m * sizeof(double));
      free_bytes(Td[k], m * sizeof(double));
    }
    for (size_t b = 0; b < B; ++b) free_bytes(ab[b], 2 * m * sizeof(double));
    for (cplx* p : cls) free_vec(p, n);
  }
}

// A cell that is its own mirror image along x and y splits into four parity
// classes of a quarter of the order each (fold.cu): an eigen-decomposition costs
// a sixteenth of the operations.  A pillar's raster is symmetric unless a pixel
// centre lies within rounding of the rim (checked on the device, sample by
// sample); a grid, a pixel raster or a planar section is where its coordinates
// are, to rounding, and its table is, exactly (CellSpec::mirrored, here at three
// heights and again at every sample).  Every other structure, and a cell found
// asymmetric on the way, takes the general way.  Below nine harmonics there is
// nothing to split.  General / folded: one 7 x 7-order pillar 38 / 11 ms, 16 at
// 11 x 11 orders 348 / 71, 16 slices of two at 13 x 9 orders 59 / 9, a taper of
// 41 orders 24.7 / 14.9, a planar taper of 11 x 5 orders 16.4 / 12.4.  Plain solves
// of a few small cells that return blocks, whose end media are solved once more
// at full order, lose up to 0.9 ms: one differential slice at 3 x 3 orders 1.3 / 1.8,
// at 7 x 7 4.6 / 5.1, at 41 3.9 / 4.8, one RCWA slice at 3 x 3 1.8 / 2.0.  On a square
// lattice the modes of two classes are degenerate in pairs; apart in their
// classes, the adaptive tree no longer depends on how a solver's rounding mixes
// them.
static bool mirror_symmetric(const CellSpec& c) {
  if (c.m() < 9 || std::getenv("VRC_NO_FOLD")) return false;
  if (c.kind == GEOM_PILLAR) return !c.pml;
  return c.mirrored(c.z0) && c.mirrored(0.5 * (c.z0 + c.z1)) && c.mirrored(c.z1);
}

namespace {
struct Held {  // device blocks of solves, given back also on errors
  Engine& E;
  std::vector<CellResult> r;
  ~Held() {
    for (auto& x : r) E.release_result(x);
  }
};
// Status of a cell from those of its classes; false: not symmetric after all
// (its classes then have no blocks).
bool class_status(const std::vector<CellResult>& r, size_t i, int* status) {
  *status = ST_OK;
  for (int k = 0; k < 4; ++k) {
    const int s = r[4 * i + k].status;
    if (s == ST_ASYMMETRIC) return false;
    if (s && !*status) *status = s;
  }
  return true;
}
void copy_counts(CellResult& r, const CellResult& from, int status) {
  r.status = status;
  r.N = from.N;
  r.n_eig = from.n_eig;
  r.n_samples = from.n_samples;
  r.n_nodes = from.n_nodes;
  r.nodes = from.nodes;
}
}  // namespace

void Engine::solve(const std::vector<CellSpec>& cells, int method, const RedhefferOpts& o, int nslices,
                   std::vector<CellResult>& out, int folded) {
  if (method == 0) {
    RedhefferOpts ro = o;
    ro.folded = folded;
    redheffer(cells, ro, out);
  } else if (method == 1) {
    rcwa(cells, nslices, out, folded);
  } else {
    differential(cells, nslices, out, folded);
  }
}

// The classes' S-matrices in the modes of the full-order end media, which are
// solved as ever, so that modes keep their order and phases: each class's
// blocks go over to its Fourier basis (W1 Tuu W0^-1 ...), those add up to the
// full one, and that goes over to the end modes.
void Engine::unfold_results(const std::vector<CellSpec>& cells, const std::vector<CellResult>& sub,
                            const std::vector<int>& pick, std::vector<CellResult>& out) {
  std::map<std::pair<int, int>, std::vector<int>> by_shape;
  for (int i : pick) by_shape[{cells[i].nx, cells[i].ny}].push_back(i);
  for (auto& kv : by_shape) {
    const int nx = kv.first.first, ny = kv.first.second, n = 2 * nx * ny, d = solved_order(n, FOLD_ALL);
    const std::vector<int>& ids = kv.second;
    const size_t B = ids.size();
    // end media at full order
    std::vector<CellDev*> cds;
    std::vector<SampleReq> sr;
    std::vector<EigReq> er;
    for (int i : ids) {
      const CellSpec& s = cells[i];
      CellResult& r = out[i];
      r.n = n;
      cds.push_back(prepare_cell(s));
      for (cplx** p : {&r.W0, &r.V0, &r.W0inv, &r.W1, &r.V1, &r.W1inv, &r.Tdd, &r.Tuu, &r.Rud, &r.Rdu}) *p = mat(n);
      r.gam0 = vec(n);
      r.gam1 = vec(n);
      for (int e = 0; e < 2; ++e) {
        const bool has = e ? s.has_end1 : s.has_end0;
        sr.push_back({&s, cds.back(), has ? s.z0 : (e ? s.z1 : s.z0), has, e ? s.eps_end1 : s.eps_end0, mat(n), mat(n)});
        er.push_back({sr.back().P, sr.back().Q, e ? r.W1 : r.W0, e ? r.V1 : r.V0, e ? r.W1inv : r.W0inv, nullptr,
                      e ? r.gam1 : r.gam0});
      }
    }
    std::vector<int> ast, est;
    assemble(sr, &ast);
    eig(er, n, &est);
    for (size_t q = 0; q < 2 * B; ++q) {
      const int s = q < ast.size() && ast[q] ? ast[q] : (q < est.size() ? est[q] : 0);
      if (s && !out[ids[q / 2]].status) out[ids[q / 2]].status = s;
    }
    for (auto& r : sr) {
      free_mat(r.P, n);
      free_mat(r.Q, n);
    }
    for (auto* cd : cds) release_cell(cd);
    // per block (Tdd, Tuu, Rud, Rdu): out-side and in-side ends
    const int oe[4] = {0, 1, 1, 0}, ie[4] = {1, 0, 1, 0};
    std::vector<cplx*> tmp, F, T;  // d x d products, n x n Fourier blocks and products
    std::vector<GemmDesc> g1, g2, h1, h2;
    std::vector<UnfoldMatDesc> ud;
    for (size_t b = 0; b < B; ++b) {
      const CellResult* c = &sub[4 * ids[b]];
      CellResult& r = out[ids[b]];
      cplx* const full[4] = {r.Tdd, r.Tuu, r.Rud, r.Rdu};
      for (int q = 0; q < 4; ++q) {
        UnfoldMatDesc u;
        for (int k = 0; k < 4; ++k) {
          const cplx* blk = q == 0 ? c[k].Tdd : q == 1 ? c[k].Tuu : q == 2 ? c[k].Rud : c[k].Rdu;
          cplx *t = mat(d), *f = mat(d);
          tmp.push_back(t);
          tmp.push_back(f);
          g1.push_back({oe[q] ? c[k].W1 : c[k].W0, blk, t, nullptr, nullptr, nullptr});
          g2.push_back({t, ie[q] ? c[k].W1inv : c[k].W0inv, f, nullptr, nullptr, nullptr});
          u.in[k] = f;
        }
        F.push_back(mat(n));
        T.push_back(mat(n));
        u.out = F.back();
        ud.push_back(u);
        h1.push_back({oe[q] ? r.W1inv : r.W0inv, F.back(), T.back(), nullptr, nullptr, nullptr});
        h2.push_back({T.back(), ie[q] ? r.W1 : r.W0, full[q], nullptr, nullptr, nullptr});
      }
    }
    gemm(g1, d, mk(1, 0), mk(0, 0), 0.0);
    gemm(g2, d, mk(1, 0), mk(0, 0), 0.0);
    {
      Prof pr(*this, "elementwise", 0.0, 80.0 * n * (double)n * ud.size());
      unfold_matrices(upload(ud), (int)ud.size(), nx, ny, stream_);
    }
    gemm(h1, n, mk(1, 0), mk(0, 0), 0.0);
    gemm(h2, n, mk(1, 0), mk(0, 0), 0.0);
    sync();
    for (auto* p : tmp) free_mat(p, d);
    for (auto* p : F) free_mat(p, n);
    for (auto* p : T) free_mat(p, n);
  }
}

void Engine::solve_cells(const std::vector<CellSpec>& cells, int method, const RedhefferOpts& o, int nslices,
                         std::vector<CellResult>& out) {
  for (const auto& c : cells) validate(c);
  std::vector<int> general, mirrored;
  for (size_t c = 0; c < cells.size(); ++c) (mirror_symmetric(cells[c]) ? mirrored : general).push_back((int)c);
  if (mirrored.empty()) {
    solve(cells, method, o, nslices, out, FOLD_NONE);
    return;
  }
  start_results(cells, out);
  {
    std::vector<CellSpec> one, four;
    for (int c : mirrored) {
      one.push_back(cells[c]);
      four.insert(four.end(), 4, cells[c]);
    }
    Held h{*this, {}}, full{*this, {}};
    solve(four, method, o, nslices, h.r, FOLD_ALL);
    start_results(one, full.r);
    std::vector<int> pick;
    for (size_t i = 0; i < mirrored.size(); ++i) {
      int status;
      if (class_status(h.r, i, &status)) {
        copy_counts(full.r[i], h.r[4 * i], status);
        pick.push_back((int)i);
      } else {
        general.push_back(mirrored[i]);
      }
    }
    unfold_results(one, h.r, pick, full.r);
    for (int i : pick) {
      out[mirrored[i]] = full.r[i];
      full.r[i] = CellResult();
    }
  }
  if (general.empty()) return;
  std::sort(general.begin(), general.end());
  std::vector<CellSpec> cs;
  for (int c : general) cs.push_back(cells[c]);
  std::vector<CellResult> g;
  solve(cs, method, o, nslices, g, FOLD_NONE);
  for (size_t i = 0; i < general.size(); ++i) out[general[i]] = g[i];
}

void Engine::solve_powers(const std::vector<CellSpec>& cells, int method, const RedhefferOpts& o, int nslices,
                          int side, int flux_norm, std::vector<CellResult>& res, std::vector<std::vector<double>>& R,
                          std::vector<std::vector<double>>& T) {
  for (const auto& c : cells) validate(c);
  start_results(cells, res);
  R.assign(cells.size(), {});
  T.assign(cells.size(), {});
  std::vector<int> general, mirrored;
  for (size_t c = 0; c < cells.size(); ++c)
    (mirror_symmetric(cells[c]) && cells[c].has_end0 && cells[c].has_end1 ? mirrored : general).push_back((int)c);
  if (!mirrored.empty()) {
    std::vector<CellSpec> one, four;
    for (int c : mirrored) {
      one.push_back(cells[c]);
      four.insert(four.end(), 4, cells[c]);
    }
    Held h{*this, {}};
    solve(four, method, o, nslices, h.r, FOLD_EXCITED);
    std::vector<int> pick;
    std::vector<CellSpec> ps;
    std::vector<CellResult> pr;  // (h keeps the blocks)
    for (size_t i = 0; i < mirrored.size(); ++i) {
      int status;
      if (!class_status(h.r, i, &status)) {
        general.push_back(mirrored[i]);
        continue;
      }
      copy_counts(res[mirrored[i]], h.r[4 * i], status);
      pick.push_back(mirrored[i]);
      ps.push_back(one[i]);
      pr.insert(pr.end(), h.r.begin() + 4 * i, h.r.begin() + 4 * i + 4);
    }
    std::vector<std::vector<double>> Rm, Tm;
    order_powers(ps, pr, side, flux_norm, Rm, Tm, FOLD_EXCITED);
    for (size_t i = 0; i < pick.size(); ++i) {
      R[pick[i]] = std::move(Rm[i]);
      T[pick[i]] = std::move(Tm[i]);
    }
  }
  if (general.empty()) return;
  std::sort(general.begin(), general.end());
  std::vector<CellSpec> cs;
  for (int c : general) cs.push_back(cells[c]);
  Held h{*this, {}};
  solve(cs, method, o, nslices, h.r, FOLD_NONE);
  std::vector<std::vector<double>> Rg, Tg;
  order_powers(cs, h.r, side, flux_norm, Rg, Tg);
  for (size_t i = 0; i < general.size(); ++i) {
    const int c = general[i];
    R[c] = std::move(Rg[i]);
    T[c] = std::move(Tg[i]);
    copy_counts(res[c], h.r[i], h.r[i].status);
  }
}

}  // namespace vrc
