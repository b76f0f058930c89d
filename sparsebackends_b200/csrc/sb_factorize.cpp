// Block factorisations of SparseBackends (src/ops_factorize.jl) on the device.
//
// blocksparse_left_qr (ops_factorize.jl:8-43): A[(l, r) | s] -> M with
//   M[(li-1)*d_s + s, ri] = A[l_vals[li], r_vals[ri]][s] over the sorted distinct
//   l and r values of the keys, thin QR M = Q R (k = min(rows, cols)), and
//   Q as a block-sparse tensor (l | s, b) with one block for every l value
//   (setindex! creates it, storage.jl:114-124).  Householder QR on the device.
// blocksparse_svd (ops_factorize.jl:50-148): A[(L, R) | s1, s2] grouped by L;
//   per group M_L = [A[L, R_1] ... A[L, R_n]] as d_s1 x (n * d_s2), SVD of every
//   group (batched one-sided Jacobi, one CTA per group), then the global
//   truncation: singular values sorted decreasing (stable), keep
//   min(maxdim, total), then drop while count > mindim and sv < cutoff*max_sv,
//   truncerr = sum of the dropped sv^2; per group the first k_kept columns,
//   new bond indices contiguous per group in L order; U blocks (L, nb) =
//   U_L[:, col] (times sv when ortho = right), SV blocks (nb, R_j) =
//   Vt_L[col, R_j part] (times sv when ortho = left).
// The index bookkeeping (distinct values, groups, the sort of the singular
// values and the keep counts) is host work, as in the reference; every value
// is computed on the device.
#include <algorithm>
#include <numeric>

#include "sb_internal.hpp"
#include "sb_kernels.hpp"

namespace sb {

namespace {

void gather(Ctx* ctx, const double* src, double* dst, const double* scale, const std::vector<Gather2D>& items) {
  if (items.empty()) return;
  int64_t mx = 0;
  for (const auto& it : items) mx = std::max(mx, it.rows * it.cols);
  DevBuf d = upload(ctx, items);
  ProfScope ps(ctx, PROF_OTHER, 0.0, 0.0);
  SB_CK(launch_gather_2d(src, dst, scale, d.as<Gather2D>(), static_cast<int64_t>(items.size()), mx, ctx->stream));
  ctx->note_launch();
}

// The sorted distinct values of one prefix axis and the position of each:
// by a table over the axis when it is not much longer than the key list
// (two passes over the keys), else by sorting.
struct Ranks {
  std::vector<int64_t> vals, table;  // table[x] = position of value x, when used
  Ranks(const Tensor& A, int axis) {
    const int64_t d = A.dims[axis];
    if (d <= 4 * A.nkeys + 1024) {
      table.assign(d + 1, -1);
      for (int64_t i = 0; i < A.nkeys; ++i) table[A.key(i)[axis]] = 0;
      for (int64_t x = 1; x <= d; ++x)
        if (table[x] == 0) {
          table[x] = static_cast<int64_t>(vals.size());
          vals.push_back(x);
        }
      return;
    }
    for (int64_t i = 0; i < A.nkeys; ++i) vals.push_back(A.key(i)[axis]);
    std::sort(vals.begin(), vals.end());
    vals.erase(std::unique(vals.begin(), vals.end()), vals.end());
  }
  int64_t of(int64_t x) const {
    if (!table.empty()) return table[x];
    return static_cast<int64_t>(std::lower_bound(vals.begin(), vals.end(), x) - vals.begin());
  }
};

}  // namespace

QrResult blocksparse_left_qr(Ctx* ctx, const Tensor& A) {
  require(A.kind == BS, SB_ERR_UNSUPPORTED_TYPES, "blocksparse_left_qr: block-sparse tensor expected");
  require(A.N() == 3 && A.n2 == 1, SB_ERR_UNSUPPORTED_LAYOUT,
          "blocksparse_left_qr: expects N = 3 with prefix (l, r) and dense tail (s)");
  require_uniform(A, "blocksparse_left_qr");
  require(A.nkeys > 0, SB_ERR_INVALID_ARG, "blocksparse_left_qr: tensor has no blocks");
  QrResult out;
  Ranks lr(A, 0), rr(A, 1);
  out.l_vals = lr.vals;
  out.r_vals = rr.vals;
  const int64_t ds = A.dims[2];
  const int64_t nl = static_cast<int64_t>(out.l_vals.size()), nr = static_cast<int64_t>(out.r_vals.size());
  const int64_t m = nl * ds, n = nr, k = std::min(m, n);
  // dense M (column-major m x n)
  DevBuf M(ctx, std::max<int64_t>(m * n, 1) * sizeof(double));
  if (m * n) SB_CK(cudaMemsetAsync(M.raw(), 0, m * n * sizeof(double), ctx->stream));
  std::vector<int64_t> so(A.nkeys), dof(A.nkeys), ln(A.nkeys, ds);
  for (int64_t i = 0; i < A.nkeys; ++i) {
    so[i] = A.block_off(i);
    dof[i] = lr.of(A.key(i)[0]) * ds + rr.of(A.key(i)[1]) * m;
  }
  copy_blocks(ctx, A.data.d(), M.d(), so, dof, ln);
  DevBuf tau(ctx, std::max<int64_t>(householder_scalars(m, n), 1) * sizeof(double));
  DevBuf Q(ctx, std::max<int64_t>(m * k, 1) * sizeof(double));
  if (k > 0) {
    ProfScope ps(ctx, PROF_OTHER, 4.0 * m * n * k, 8.0 * m * n);
    int64_t launches = 0;
    SB_CK(launch_householder_qr(M.d(), m, n, tau.d(), ctx->stream, &launches));
    SB_CK(launch_householder_form_q(M.d(), m, k, tau.d(), Q.d(), ctx->stream, &launches));
    ctx->note_launch(launches);
  }
  // R (k x n) dense
  out.R = make_tensor(ctx, DENSE, {k, n}, 2);
  out.R->data = DevBuf(ctx, std::max<int64_t>(k * n, 1) * sizeof(double));
  if (k * n) {
    SB_CK(launch_upper(M.d(), m, k, n, out.R->data.d(), ctx->stream));
    ctx->note_launch();
  }
  // Q as block-sparse (l | s, b): one block per l value, ds x k each
  out.Q = make_tensor(ctx, BS, {A.dims[0], ds, k}, 2);
  std::vector<Gather2D> items;
  for (int64_t li = 0; li < nl && k > 0; ++li) {
    out.Q->keys.push_back(out.l_vals[li]);
    items.push_back(Gather2D{li * ds, li * ds * k, ds, k, 1, m, 1, ds, -1});
  }
  out.Q->nkeys = static_cast<int64_t>(items.size());
  out.Q->data = DevBuf(ctx, std::max<int64_t>(out.Q->nkeys * ds * k, 1) * sizeof(double));
  gather(ctx, Q.d(), out.Q->data.d(), nullptr, items);
  return out;
}

SvdResult blocksparse_svd(Ctx* ctx, const Tensor& A, bool ortho_right, int64_t maxdim, int64_t mindim,
                          double cutoff) {
  require(A.kind == BS, SB_ERR_UNSUPPORTED_TYPES, "blocksparse_svd: block-sparse tensor expected");
  require(A.N() == 4 && A.n2 == 2, SB_ERR_UNSUPPORTED_LAYOUT,
          "blocksparse_svd: expects N = 4 with prefix (L, R) and dense tail (s1, s2)");
  require_uniform(A, "blocksparse_svd");
  const int64_t nL = A.dims[0], nR = A.dims[1], d1 = A.dims[2], d2 = A.dims[3];
  require(d1 <= kSvdMaxRows, SB_ERR_UNSUPPORTED_LAYOUT, "blocksparse_svd: first dense dim exceeds 32");
  require(A.nkeys > 0, SB_ERR_INVALID_ARG, "blocksparse_svd: tensor has no blocks");
  require(maxdim >= 1 && mindim >= 0 && cutoff >= 0.0, SB_ERR_INVALID_ARG,
          "blocksparse_svd: maxdim >= 1, mindim >= 0, cutoff >= 0 required");
  // group keys by L (keys are sorted by L + nL*R, so R ascends within a group)
  const Ranks lr(A, 0);
  struct G {
    int64_t L, n, a_off, u_off, s_off, k;
  };
  std::vector<G> gs(lr.vals.size());
  std::vector<int64_t> gof(A.nkeys), col(A.nkeys);  // group of key i, its place in the group
  for (int64_t i = 0; i < A.nkeys; ++i) {
    gof[i] = lr.of(A.key(i)[0]);
    col[i] = gs[gof[i]].n++;
  }
  int64_t aw = 0, uw = 0, sw = 0;
  for (size_t gi = 0; gi < gs.size(); ++gi) {
    const int64_t n = gs[gi].n * d2;
    gs[gi] = G{lr.vals[gi], n, aw, uw, sw, std::min(d1, n)};
    aw += d1 * n;
    uw += d1 * d1;
    sw += d1;
  }
  // M_L[s1, j*d2 + s2] (row-major, row length n) = A block [s1 + s2*d1]
  std::vector<Gather2D> items(A.nkeys);
  for (int64_t i = 0; i < A.nkeys; ++i) {
    const G& g = gs[gof[i]];
    items[i] = Gather2D{A.block_off(i), g.a_off + col[i] * d2, d1, d2, 1, d1, g.n, 1, -1};
  }
  SvdResult out;
  DevBuf W(ctx, std::max<int64_t>(aw, 1) * sizeof(double)), Vt(ctx, std::max<int64_t>(aw, 1) * sizeof(double));
  DevBuf U(ctx, std::max<int64_t>(uw, 1) * sizeof(double)), S(ctx, std::max<int64_t>(sw, 1) * sizeof(double));
  gather(ctx, A.data.d(), W.d(), nullptr, items);
  std::vector<double> sv(sw);
  if (!gs.empty()) {
    std::vector<SvdGroup> sg;
    for (const G& g : gs) sg.push_back(SvdGroup{g.a_off, g.n, g.u_off, g.s_off, static_cast<int32_t>(d1), 0});
    DevBuf dg = upload(ctx, sg);
    DevBuf st(ctx, sizeof(int));
    SB_CK(cudaMemsetAsync(st.raw(), 0, sizeof(int), ctx->stream));
    {
      ProfScope ps(ctx, PROF_OTHER, 0.0, 16.0 * aw);
      SB_CK(launch_svd_rows(W.d(), Vt.d(), U.d(), S.d(), dg.as<SvdGroup>(), static_cast<int64_t>(sg.size()), 64,
                            st.as<int>(), ctx->stream));
    }
    ctx->note_launch();
    require(download<int>(ctx, st.raw(), 1)[0] == 0, SB_ERR_ASSERTION,
            "blocksparse_svd: Jacobi SVD did not converge in 64 sweeps");
    sv = download<double>(ctx, S.raw(), sw);
  }
  // global truncation (host bookkeeping on the singular values)
  struct SvRef {
    double sv;
    int64_t g, col;
  };
  std::vector<SvRef> all;
  for (size_t gi = 0; gi < gs.size(); ++gi)
    for (int64_t c = 0; c < gs[gi].k; ++c) all.push_back(SvRef{sv[gs[gi].s_off + c], static_cast<int64_t>(gi), c});
  std::stable_sort(all.begin(), all.end(), [](const SvRef& a, const SvRef& b) { return a.sv > b.sv; });
  const double max_sv = all.empty() ? 1.0 : all[0].sv;
  int64_t keep = std::min<int64_t>(maxdim, static_cast<int64_t>(all.size()));
  while (keep > mindim && all[keep - 1].sv < cutoff * max_sv) --keep;
  out.truncerr = 0.0;
  for (size_t i = static_cast<size_t>(keep); i < all.size(); ++i) out.truncerr += all[i].sv * all[i].sv;
  std::vector<int64_t> kk(gs.size(), 0), off(gs.size(), 0);
  for (int64_t i = 0; i < keep; ++i) ++kk[all[i].g];
  int64_t nb = 0;
  for (size_t gi = 0; gi < gs.size(); ++gi) {
    off[gi] = nb;
    nb += kk[gi];
  }
  out.svs.assign(nb, 0.0);
  // U: dims (nL, nb, d1), prefix (L, b), dense s1; keys in nb order are sorted
  out.U = make_tensor(ctx, BS, {nL, nb, d1}, 1);
  out.SV = make_tensor(ctx, BS, {nb, nR, d2}, 1);
  std::vector<Gather2D> ui, vg(A.nkeys);
  out.U->keys.reserve(2 * nb);
  for (size_t gi = 0; gi < gs.size(); ++gi) {
    const G& g = gs[gi];
    for (int64_t c = 0; c < kk[gi]; ++c) {
      out.svs[off[gi] + c] = sv[g.s_off + c];
      out.U->keys.push_back(g.L);
      out.U->keys.push_back(off[gi] + c + 1);
    }
    if (kk[gi] > 0)  // column c of U_L, times its singular value when ortho = right
      ui.push_back(Gather2D{g.u_off, off[gi] * d1, d1, kk[gi], 1, d1, 1, d1, ortho_right ? g.s_off : -1});
  }
  out.U->nkeys = nb;
  out.U->data = DevBuf(ctx, std::max<int64_t>(nb * d1, 1) * sizeof(double));
  gather(ctx, U.d(), out.U->data.d(), S.d(), ui);
  // SV's keys (b, R) column-major: A's keys run through R, and for one R
  // through L, whose bond values b ascend with it
  int64_t nsv = 0;
  for (int64_t i = 0; i < A.nkeys; ++i) nsv += kk[gof[i]];
  out.SV->keys.resize(2 * nsv);
  int64_t at = 0;
  for (int64_t i = 0; i < A.nkeys; ++i) {
    const int64_t gi = gof[i], R = A.key(i)[1];
    const G& g = gs[gi];
    vg[i] = Gather2D{g.a_off + col[i] * d2, at * d2, d2, kk[gi], 1, g.n, 1, d2, ortho_right ? -1 : g.s_off};
    for (int64_t c = 0; c < kk[gi]; ++c, ++at) {
      out.SV->keys[2 * at] = off[gi] + c + 1;
      out.SV->keys[2 * at + 1] = R;
    }
  }
  out.SV->nkeys = nsv;
  out.SV->data = DevBuf(ctx, std::max<int64_t>(nsv * d2, 1) * sizeof(double));
  gather(ctx, Vt.d(), out.SV->data.d(), S.d(), vg);
  return out;
}

}  // namespace sb
