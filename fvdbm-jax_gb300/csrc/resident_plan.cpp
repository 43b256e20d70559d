// Host tables of the resident steps: the cells are cut into compact parts, one
// per thread block, and every index a block uses during a run of steps becomes
// local to it: its own cells, then the halo cells it imports from other blocks,
// then one ghost entry per ghost face (resident.cu); in place (resident_in_place.cu)
// the interior cells in the order of the sweep, and rows for what the others read.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <future>
#include <system_error>

#include "fvdbm_internal.h"

namespace fvdbm {

namespace {

// Threads for a mesh of N cells: one for every so many, the caller among them.  ms of a plan on 16
// host cores, one thread / these: 12k cells 1.7 / 0.9, 20k 2.5 / 1.3, 60k 6.3 / 2.3, 250k 20.0 (most
// of it on one) / 8.7; a thread for every 1,500 or 6,000 cells 1.0 and 1.4 at 12k.
constexpr int THREAD_CELLS = 3000, THREADS = 8;
int threads_for(int N) { return std::max(1, std::min(THREADS, N / THREAD_CELLS)); }

struct Point {
  float x[2];
  int32_t id;
};

// Recursive bisection of pts[a, b) (device cells) into parts [p0, p0 + parts)
// of equal size, each cut across the longer side of its bounding box: compact
// parts keep the halos short.  Without coordinates the device order is cut.
void bisect(bool xy, std::vector<Point>& pts, int a, int b, int p0, int parts, std::vector<int32_t>& part_end,
            int many) {
  if (parts == 1) {
    part_end[p0] = b;
    return;
  }
  const int left = parts / 2;
  const int mid = a + int(int64_t(b - a) * left / parts);
  if (xy) {
    float lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
    for (int i = a; i < b; ++i)
      for (int d = 0; d < 2; ++d) {
        lo[d] = std::min(lo[d], pts[i].x[d]);
        hi[d] = std::max(hi[d], pts[i].x[d]);
      }
    const int d = hi[0] - lo[0] >= hi[1] - lo[1] ? 0 : 1;
    std::nth_element(pts.begin() + a, pts.begin() + mid, pts.begin() + b, [d](const Point& u, const Point& v) {
      return u.x[d] != v.x[d] ? u.x[d] < v.x[d] : u.id < v.id;
    });
  }
  std::future<void> other;  // (a large part's halves side by side)
  try {
    if (b - a > many)
      other = std::async(std::launch::async, [&] { bisect(xy, pts, a, mid, p0, left, part_end, many); });
  } catch (const std::system_error&) {
  }
  bisect(xy, pts, mid, b, p0 + left, parts - left, part_end, many);
  if (other.valid())
    other.get();
  else
    bisect(xy, pts, a, mid, p0, left, part_end, many);
}

// Cells of a chunk of the sweep: chunks of equal size, at most a cell per thread.
int chunk_cells(int inner, int threads) {
  const int n = std::max(1, (inner + threads - 1) / threads);
  return std::max(32, ((inner + n - 1) / n + 31) / 32 * 32);
}

// f(t, scratch) of every block, by a few threads (by fewer when there are none to be
// had), each with its own make().
template <class M, class F>
void for_blocks(int N, int B, const M& make, const F& f) {
  const int n = threads_for(N);
  auto run = [&](int i) {
    auto scratch = make();
    for (int t = i; t < B; t += n) f(t, scratch);
  };
  std::vector<std::future<void>> work;
  for (int i = 1; i < n && i < B; ++i) {
    try {
      work.push_back(std::async(std::launch::async, run, i));
    } catch (const std::system_error&) {
      run(i);
    }
  }
  run(0);
  for (auto& w : work) w.get();
}
template <class F>
void for_blocks(int N, int B, const F& f) {
  for_blocks(N, B, [] { return 0; }, [&](int t, int) { f(t); });
}

// Tables of one block, before they are joined: indices into themselves.
struct BlockTables {
  std::vector<int32_t> halo_dev, halo_exp, st_loc, halo_st, nd, fz_dev, gh;
  std::vector<uint32_t> en_st;
  std::vector<float> nd_sw, en_w;
  bool usable = true;
  int rows = 0, stride = 0;
  void clear() {
    for (auto* v : {&halo_dev, &halo_exp, &st_loc, &halo_st, &nd, &fz_dev, &gh}) v->clear();
    en_st.clear();
    nd_sw.clear();
    en_w.clear();
    usable = true;
  }
};

// Order of the update in place: the interior cells, the first `inner` of the
// part's n, along the longer side of its bounding box, in chunks of TC.  Within
// a chunk the device order (coalesced reads and writes of the state).
void sweep_order(const float* xy, const HostPlan& hp, int32_t* ids, int n, int inner, int TC) {
  if (!xy) return;
  float lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
  std::vector<Point> pts(n);
  for (int i = 0; i < n; ++i) {
    const size_t c = size_t(hp.cell_old[ids[i]]);
    pts[i] = Point{{xy[2 * c], xy[2 * c + 1]}, ids[i]};
    for (int d = 0; d < 2; ++d) {
      lo[d] = std::min(lo[d], pts[i].x[d]);
      hi[d] = std::max(hi[d], pts[i].x[d]);
    }
  }
  const int d = hi[0] - lo[0] >= hi[1] - lo[1] ? 0 : 1;
  std::sort(pts.begin(), pts.begin() + inner, [d](const Point& u, const Point& v) {
    return u.x[d] != v.x[d] ? u.x[d] < v.x[d] : u.id < v.id;
  });
  for (int i = 0; i < inner; ++i) ids[i] = pts[i].id;
  for (int i = 0; i < inner; i += TC) std::sort(ids + i, ids + std::min(inner, i + TC));
}

}  // namespace

void build_resident(const fvdbm_mesh_t& m, const fvdbm_params_t& pr, const HostPlan& hp, int n_blocks,
                    const float* case_dt, bool in_place, ResidentPlan& rp) {
  rp = ResidentPlan{};
  rp.in_place = in_place;
  const int N = hp.N, H = hp.hrows;
  if (N == 0 || !hp.fusable || hp.K != 3 || n_blocks < 1) return;
  // the kernel drops terms that are +-0 for finite geometry
  auto f32 = [](uint32_t u) {
    float x;
    std::memcpy(&x, &u, 4);
    return x;
  };
  const int G = int(hp.hf.size() / (size_t(H) * 32)), share_of = 256;  // groups of 32 cells, by 256
  std::vector<char> finite((G + share_of - 1) / share_of, 1);
  for_blocks(N, int(finite.size()), [&](int t) {
    uint32_t most = 0;  // (all exponent bits set: not finite)
    for (int g = t * share_of; g < std::min(G, (t + 1) * share_of); ++g) {
      const uint32_t* w = hp.hf.data() + size_t(g) * H * 32;
      for (int i = 3 * 32; i < H * 32; ++i) most = std::max(most, w[i] & 0x7f800000u);
    }
    finite[t] = most != 0x7f800000u;
  });
  for (char ok : finite)
    if (!ok) return;
  for (float a : hp.inv_area)
    if (!std::isfinite(a)) return;
  const bool lw = hp.scheme == FVDBM_LAX_WENDROFF, sc = hp.variant == FVDBM_VARIANT_FACE_SCALE;
  const int NP = hp.q == 13 ? 6 : 4;
  const int R = hp.fast ? H : 3 * ((lw ? 5 + NP : 4) + (sc ? 1 : 0));
  if (in_place && (hp.q != 9 || lw || sc)) return;
  const float* xy = m.cell_xy;
  for (int64_t i = 0; xy && i < 2 * int64_t(N); ++i)
    if (!std::isfinite(xy[i])) xy = nullptr;
  auto hfi = [&](int i, int row) { return size_t(i >> 5) * size_t(H) * 32 + size_t(row) * 32 + (i & 31); };

  // ---- parts: those of a batch's case stay inside it, its share of the blocks
  // by its cells (at least one; the cases with the most cells per block first)
  const int B = std::min(n_blocks, N), S = std::max(1, hp.S);
  if (S > B) return;
  std::vector<int32_t> case_cell = hp.S ? hp.case_cell : std::vector<int32_t>{0, N}, share(S, 1);
  for (int left = B - S; left > 0; --left) {
    int best = -1;
    double most = 1.0;
    for (int s = 0; s < S; ++s) {
      const double per = double(case_cell[s + 1] - case_cell[s]) / share[s];
      if (per > most) {
        most = per;
        best = s;
      }
    }
    if (best < 0) return;
    ++share[best];
  }
  std::vector<int32_t> ids(N), part_end(B), part(N), loc(N);
  {
    std::vector<Point> pts(N);
    for (int i = 0; i < N; ++i) {
      const int32_t c = hp.cell_old[i];
      pts[i] = Point{{xy ? xy[2 * size_t(c)] : 0.0f, xy ? xy[2 * size_t(c) + 1] : 0.0f}, i};
    }
    for (int s = 0, p0 = 0; s < S; p0 += share[s++])
      bisect(xy != nullptr, pts, case_cell[s], case_cell[s + 1], p0, share[s], part_end,
             std::max(THREAD_CELLS, N / THREADS));
    for (int i = 0; i < N; ++i) ids[i] = pts[i].id;
  }
  for (int t = 0, i = 0; t < B; ++t)
    for (; i < part_end[t]; ++i) part[ids[i]] = t;

  // ---- what each block imports: the cells across its faces and the stencil
  // cells of the boundary nodes its ghost faces read.  A node that no ghost
  // face reads belongs to the block of its first stencil cell.
  std::vector<std::vector<int32_t>> imp(B), nodes(B);
  std::vector<std::vector<int32_t>> ghost_cells(B);
  std::vector<char> node_used(hp.M, 0);
  for (size_t g = 0; g < hp.gh_a.size(); ++g) node_used[hp.gh_a[g]] = node_used[hp.gh_b[g]] = 1;
  std::vector<std::vector<int32_t>> extra(B);
  for (int d = 0; d < hp.Mc; ++d)
    if (!node_used[d])
      extra[hp.nd_ptr[d + 1] > hp.nd_ptr[d] ? part[hp.nd_cell[hp.nd_ptr[d]] & ~ND_NEQ_ZERO] : 0].push_back(d);
  std::vector<char> links(size_t(B) * B, 0);  // links[t * B + u]: t imports from u
  const auto no_node = [&] { return std::vector<int32_t>(hp.M, -1); };
  for_blocks(N, B, no_node, [&](int t, std::vector<int32_t>& nmark) {
    auto need = [&](int32_t c) {
      if (part[c] != t) {
        imp[t].push_back(c);
        links[size_t(t) * B + part[c]] = 1;
      }
    };
    auto node = [&](int32_t d) {
      if (nmark[d] == t) return;
      nmark[d] = t;
      nodes[t].push_back(d);
      if (d >= hp.Mc) return;
      for (int e = hp.nd_ptr[d]; e < hp.nd_ptr[d + 1]; ++e) need(int32_t(hp.nd_cell[e] & ~ND_NEQ_ZERO));
      if (hp.nd_npad[d] > 0) need(hp.last_cell_new);
    };
    for (int i = t ? part_end[t - 1] : 0; i < part_end[t]; ++i)
      for (int k = 0; k < 3; ++k) {
        const int32_t code = int32_t(hp.hf[hfi(ids[i], k)]);
        if (code & HF_GHOST) {
          node(hp.gh_a[code >> HF_SHIFT]);
          node(hp.gh_b[code >> HF_SHIFT]);
        } else {
          need(code >> HF_SHIFT);
        }
      }
    for (int32_t d : extra[t]) node(d);
    std::sort(imp[t].begin(), imp[t].end());
    imp[t].erase(std::unique(imp[t].begin(), imp[t].end()), imp[t].end());
  });
  // a block may overwrite an exported value only once its reader has moved
  // on, which it learns from the reader's own exports: every link goes both
  // ways (a one-way link gets one cell to read back)
  for (int t = 0; t < B; ++t)
    for (int u = 0; u < B; ++u)
      if (links[size_t(t) * B + u] && !links[size_t(u) * B + t]) {
        const int32_t c = ids[t ? part_end[t - 1] : 0];
        imp[u].push_back(c);
        links[size_t(u) * B + t] = 1;
      }

  // ---- local order: one interior cell per cell thread (work that waits for
  // nothing), then the cells with halo faces or exports, those with ghost faces, and
  // the remaining interior cells; export slots in that order
  std::vector<char> exported(N, 0);
  for (int t = 0; t < B; ++t)
    for (int32_t c : imp[t]) exported[c] = 1;
  std::vector<int32_t> slot(N, -1);
  // (an exported cell waits for the imports too: its next value overwrites
  // the one that its readers must have taken)
  std::vector<char> kind(exported);
  for (int t = 0; t < B; ++t) rp.max_own = std::max(rp.max_own, part_end[t] - (t ? part_end[t - 1] : 0));
  if (!in_place) resident_threads(rp.max_own, &rp.cell_threads, &rp.threads);
  {  // each part's cells in device order
    std::vector<int32_t> at(B, 0);
    for (int t = 1; t < B; ++t) at[t] = part_end[t - 1];
    for (int i = 0; i < N; ++i) ids[at[part[i]]++] = i;
  }
  std::vector<int> inside(B);  // interior cells
  for_blocks(N, B, [&](int t) {
    const auto first = ids.begin() + (t ? part_end[t - 1] : 0), last = ids.begin() + part_end[t];
    for (auto c = first; c != last; ++c)
      for (int k = 0; k < 3; ++k) {
        const int32_t code = int32_t(hp.hf[hfi(*c, k)]);
        if (code & HF_GHOST)
          kind[*c] = 2;
        else if (part[code >> HF_SHIFT] != t)
          kind[*c] = std::max<char>(kind[*c], 1);
      }
    const auto in_end = std::stable_partition(first, last, [&](int32_t c) { return kind[c] == 0; });
    std::stable_partition(in_end, last, [&](int32_t c) { return kind[c] == 1; });
    inside[t] = int(in_end - first);
  });
  if (in_place) {
    in_place_threads(*std::max_element(inside.begin(), inside.end()), &rp.cell_threads, &rp.threads);
    for_blocks(N, B, [&](int t) {
      const int a = t ? part_end[t - 1] : 0;
      sweep_order(xy, hp, ids.data() + a, part_end[t] - a, inside[t], chunk_cells(inside[t], rp.cell_threads));
    });
  }
  int off = 0;
  for (int t = 0; t < B; ++t) {
    const int a = t ? part_end[t - 1] : 0, b = part_end[t];
    const int inner = inside[t], TC = rp.cell_threads;
    if (!in_place && inner > TC) std::rotate(ids.begin() + a + TC, ids.begin() + a + inner, ids.begin() + b);
    ResidentBlock mb{};
    mb.own_off = off;
    mb.nown = b - a;
    mb.nin = in_place ? inner : 0;
    mb.exp_off = rp.n_export;
    mb.chunk = chunk_cells(inner, TC);
    mb.cs = hp.S ? hp.cell_case[ids[a]] : 0;
    // (the boundary cells of the update in place begin a group of 32)
    const int gap = in_place ? (inner + 31) / 32 * 32 - inner : 0;
    for (int i = a; i < b; ++i) {
      loc[ids[i]] = i - a + (i - a < inner ? 0 : gap);
      if (exported[ids[i]]) slot[ids[i]] = rp.n_export++;
    }
    off += (b - a + gap + 31) / 32 * 32;
    rp.block.push_back(mb);
  }
  rp.dev.assign(off, -1);
  if (!in_place) {  // (the ring has its classes in its order, and the slots in its codes)
    rp.exp.assign(off, -1);
    rp.cls.assign(off / 32, 0);
  }
  rp.hf.assign(size_t(off / 32) * R * 32, 0u);
  auto ri = [&](int i, int row) { return size_t(i >> 5) * size_t(R) * 32 + size_t(row) * 32 + (i & 31); };
  auto bits = [](float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
  };
  const HfRows HR{3, hp.scheme, hp.variant};
  if (hp.fv) rp.inv_area.assign(off, 0.0f);
  std::vector<int32_t> owner(hp.M, -1);  // the first block that computes the node
  for (int t = 0; t < B; ++t)
    for (int32_t d : nodes[t])
      if (owner[d] < 0) owner[d] = t;
  struct Scratch {
    std::vector<int32_t> hloc, nloc, sloc;
    BlockTables bt;  // (grown once, copied for each block)
  };
  const auto scratch = [&] {
    return Scratch{std::vector<int32_t>(N), std::vector<int32_t>(hp.M), std::vector<int32_t>(N, -1), {}};
  };
  std::vector<BlockTables> tables(B);
  for_blocks(N, B, scratch, [&](int t, Scratch& sc_) {
    auto& [hloc, nloc, sloc, bt] = sc_;
    ResidentBlock& mb = rp.block[t];
    bt.clear();
    const int a = t ? part_end[t - 1] : 0, pad = (mb.nown + 31) / 32 * 32;
    const int bnd0 = (mb.nin + 31) / 32 * 32, nb = mb.nown - mb.nin;
    std::sort(imp[t].begin(), imp[t].end(), [&](int32_t x, int32_t y) { return slot[x] < slot[y]; });
    mb.nhalo = int(imp[t].size());
    const int halo0 = in_place ? 0 : pad;
    for (int j = 0; j < mb.nhalo; ++j) {
      bt.halo_dev.push_back(imp[t][j]);
      bt.halo_exp.push_back(slot[imp[t][j]]);
      hloc[imp[t][j]] = halo0 + j;
    }
    auto local = [&](int32_t c) { return part[c] == t ? loc[c] : hloc[c]; };
    // boundary nodes: computed first, then frozen
    std::stable_partition(nodes[t].begin(), nodes[t].end(), [&](int32_t d) { return d < hp.Mc; });
    mb.last_st = 0;
    std::vector<int32_t> touched;
    // (in place: the block's own ones first)
    auto st = [&](int32_t c) {
      if (sloc[c] < 0) {
        sloc[c] = mb.nst++;
        bt.st_loc.push_back(local(c));
        touched.push_back(c);
      }
      return sloc[c];
    };
    if (in_place) {
      auto own = [&](int32_t c) {
        if (part[c] == t) st(c);
      };
      for (int32_t d : nodes[t])
        if (d < hp.Mc) {
          if (hp.nd_npad[d] > 0) own(hp.last_cell_new);
          for (int e = hp.nd_ptr[d]; e < hp.nd_ptr[d + 1]; ++e) own(int32_t(hp.nd_cell[e] & ~ND_NEQ_ZERO));
        }
      mb.nst_own = mb.nst;
    }
    for (size_t j = 0; j < nodes[t].size(); ++j) {
      const int32_t d = nodes[t][j];
      nloc[d] = int(j);
      if (d >= hp.Mc) {
        bt.fz_dev.push_back(d);
        ++mb.nf;
        continue;
      }
      ++mb.nn;
      if (hp.nd_npad[d] > 0) mb.last_st = st(hp.last_cell_new);
      bt.nd.push_back(d);
      bt.nd.push_back(hp.nd_type[d] | (hp.nd_npad[d] > 0 ? 4 : 0) | (owner[d] == t ? 8 : 0));
      bt.nd.push_back(int(bt.en_st.size()));
      bt.nd.push_back(hp.nd_ptr[d + 1] - hp.nd_ptr[d]);
      bt.nd_sw.push_back(hp.nd_sumw[d]);
      for (int e = hp.nd_ptr[d]; e < hp.nd_ptr[d + 1]; ++e) {
        const uint32_t code = hp.nd_cell[e];
        bt.en_st.push_back(uint32_t(st(int32_t(code & ~ND_NEQ_ZERO))) | (code & ND_NEQ_ZERO));
        bt.en_w.push_back(hp.nd_w[e]);
      }
    }
    for (int j = 0; in_place && j < mb.nhalo; ++j) bt.halo_st.push_back(sloc[imp[t][j]]);
    for (int32_t c : touched) sloc[c] = -1;
    mb.ne = int(bt.en_st.size());
    // face slots with local indices; ghost faces get their own entries.  In
    // place: the boundary cells' name rows, those of interior neighbours (saved)
    // and of boundary cells after the ghosts
    int ng = 0;
    for (int i = 0; in_place && i < mb.nown; ++i)
      for (int k = 0; k < 3; ++k) {
        const int32_t code = int32_t(hp.hf[hfi(ids[a + i], k)]);
        if (code & HF_GHOST) ++ng;
      }
    std::vector<int32_t> saved(in_place ? mb.nin : 0, -1);
    for (int i = mb.nin; in_place && i < mb.nown; ++i)
      for (int k = 0; k < 3; ++k) {
        const int32_t code = int32_t(hp.hf[hfi(ids[a + i], k)]), n = code >> HF_SHIFT;
        if (!(code & HF_GHOST) && part[n] == t && loc[n] < mb.nin && saved[loc[n]] < 0)
          saved[loc[n]] = mb.nsave++;
      }
    const int orow = mb.nhalo + ng, brow = orow + mb.nsave, ring = bnd0 + mb.chunk;
    // (16 bits for a neighbour, 12 for a link)
    if (in_place && (std::max(brow + nb, 9 * (ring + nb + 31)) > 0xffff || std::max(mb.nsave, nb) >= 0xfff)) bt.usable = false;
    for (int i = 0; i < mb.nown; ++i) {
      const int32_t c = ids[a + i];
      const int l = loc[c], g = mb.own_off + l;
      const bool inside = i < mb.nin;
      rp.dev[g] = c;
      if (hp.fv) rp.inv_area[g] = hp.inv_area[c];
      if (!in_place) {
        rp.exp[g] = slot[c];
        rp.cls[g / 32] = std::max<int32_t>(rp.cls[g / 32], kind[c]);
      }
      for (int row = 3; row < (hp.fast ? H : 12); ++row) rp.hf[ri(g, row)] = hp.hf[hfi(c, row)];
      if (!hp.fast)
        for (int k = 0; k < 3; ++k) {
          if (lw) {
            // the interpolation weights' quotients (xi.n * dt) / D2, in the
            // float32 operations of the per-step kernels
            rp.hf[ri(g, 12 + k)] = hp.hf[hfi(c, HR.r(k))];
            const float nx = f32(hp.hf[hfi(c, HR.nx(k))]), ny = f32(hp.hf[hfi(c, HR.ny(k))]);
            const float D2 = f32(hp.hf[hfi(c, HR.d2(k))]);
            const float v[6] = {nx, ny, nx + ny, ny - nx, 2.0f * nx, 2.0f * ny};
            for (int j = 0; j < NP; ++j) {
              const float t = (v[j] * (case_dt ? case_dt[mb.cs] : pr.delta_t)) / D2;
              if (!std::isfinite(t)) bt.usable = false;
              rp.hf[ri(g, 15 + 3 * j + k)] = bits(t);
            }
          }
          if (sc) rp.hf[ri(g, 3 * (lw ? 5 + NP : 4) + k)] = hp.hf[hfi(c, HR.sc(k))];
        }
      for (int k = 0; k < 3; ++k) {
        const int32_t code = int32_t(hp.hf[hfi(c, k)]);
        int32_t idx;
        if (code & HF_GHOST) {
          const int gi = code >> HF_SHIFT;
          int32_t rbits;
          std::memcpy(&rbits, &hp.gh_r[gi], 4);
          idx = (in_place ? mb.nhalo : pad + mb.nhalo) + mb.ng++;
          const int32_t row4[4] = {l, nloc[hp.gh_a[gi]], nloc[hp.gh_b[gi]], rbits};
          bt.gh.insert(bt.gh.end(), row4, row4 + 4);
        } else {
          const int32_t n = code >> HF_SHIFT;
          idx = local(n);
          if (inside) {
            // the sweep overwrites a chunk once the next one has been read
            if (idx < mb.nin && std::abs(idx / mb.chunk - l / mb.chunk) > 1) bt.usable = false;
            idx = idx < mb.nin ? idx : ring + idx - bnd0;  // (the boundary cells follow the ring)
            idx = (idx >> 5) * 288 + (idx & 31);
          } else if (in_place && part[n] == t) {
            idx = idx < mb.nin ? orow + saved[idx] : brow + idx - bnd0;
          }
        }
        uint32_t link = 0;
        if (in_place && k == 0) link = inside ? uint32_t(saved[i] + 1) : slot[c] < 0 ? 0u : uint32_t(slot[c] - mb.exp_off + 1);
        rp.hf[ri(g, k)] = uint32_t((code & HF_SLOT1) | (idx << HF_SHIFT)) | link << IP_LINK;
      }
    }
    bt.rows = orow + 2 * (mb.nsave + nb);
    bt.stride = in_place ? bnd0 + mb.chunk + 2 * ((nb + 31) / 32 * 32) : pad + mb.nhalo + mb.ng;
    tables[t] = bt;
  });
  // ---- the blocks' tables one after the other
  bool usable = true;
  auto join = [](auto& all, const auto& own) { all.insert(all.end(), own.begin(), own.end()); };
  for (int t = 0; t < B; ++t) {
    ResidentBlock& mb = rp.block[t];
    BlockTables& bt = tables[t];
    usable = usable && bt.usable;
    mb.halo_off = int(rp.halo_dev.size());
    mb.nd_off = int(rp.nd.size() / 4);
    mb.fz_off = int(rp.fz_dev.size());
    mb.st_off = int(rp.st_loc.size());
    mb.en_off = int(rp.en_st.size());
    mb.gh_off = int(rp.gh.size() / 4);
    mb.row_off = rp.n_rows;
    for (size_t j = 2; j < bt.nd.size(); j += 4) bt.nd[j] += mb.en_off;
    join(rp.halo_dev, bt.halo_dev);
    join(rp.halo_exp, bt.halo_exp);
    join(rp.st_loc, bt.st_loc);
    join(rp.halo_st, bt.halo_st);
    join(rp.nd, bt.nd);
    join(rp.nd_sw, bt.nd_sw);
    join(rp.en_st, bt.en_st);
    join(rp.en_w, bt.en_w);
    join(rp.fz_dev, bt.fz_dev);
    join(rp.gh, bt.gh);
    rp.n_rows += bt.rows;
    rp.stride = std::max(rp.stride, bt.stride);
    rp.max_nodes = std::max(rp.max_nodes, mb.nn + mb.nf);
    rp.max_st = std::max(rp.max_st, mb.nst);
    rp.max_table = std::max(rp.max_table, 8 * mb.nn + 4 * mb.ng + 2 * mb.ne + mb.nst + 2 * mb.nhalo);
  }
  rp.ok = usable;
}

}  // namespace fvdbm
