// Host analysis of flat SDF programs for the evaluator's exact skipping
// (sdf.cuh map): per instruction, the bounding sphere and extent of the group
// "translations, primitive, union / smooth union" that starts there; per
// left-to-right chain program, a grid of cell lists of the groups that can
// change the value inside each cell.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/myrt_cuda.h"

namespace myrt_b200 {

// Per instruction of valid programs: where a group "translations, primitive,
// union / smooth union" starts with a value already on the stack, the
// primitive's bounding sphere in the program's space (centre = summed
// translations + the primitive's own centre, radius R with distance >= |p - c|
// - R everywhere) and (absolute index after the operator, k bits). Primitives
// without such a bound (Menger sponge, degenerate parameters) and groups with a
// mirror are not skippable. Empty tables when nothing is skippable.
inline void sdf_skip_tables(myrt_sdf_view const* v, std::vector<float4>& sphere, std::vector<int2>& next) {
  sphere.assign(v->instr_count, make_float4(0.f, 0.f, 0.f, 0.f));
  next.assign(v->instr_count, make_int2(0, 0));
  std::vector<int> owner(v->instr_count, -1);
  bool any = false;
  float const* G = v->params;
  for (size_t p = 0; p < v->program_count; ++p) {
    myrt_sdf_program const pr = v->programs[p];
    int depth = 0;
    for (int g = 0; g < pr.count; ++g) {
      int const ag = pr.first + g;
      int j = g;
      double c[3] = {0.0, 0.0, 0.0};
      // a group starts at its first modifier (or at the primitive when it has
      // none): the evaluator tests the bound before applying any of them
      bool ok = depth >= 1 && (g == 0 || v->instrs[ag - 1].op < MYRT_SDF_TRANSLATE);
      while (ok && j < pr.count && v->instrs[pr.first + j].op >= MYRT_SDF_TRANSLATE) {
        myrt_sdf_instr const m = v->instrs[pr.first + j];
        if (m.op != MYRT_SDF_TRANSLATE) ok = false;
        else
          for (int a = 0; a < 3; ++a) c[a] += double(G[m.param_offset + a]);
        ++j;
      }
      double R = 0.0;
      bool bounded = false;  // only the primitives below have a bounding sphere
      if (ok && j + 1 < pr.count) {
        myrt_sdf_instr const prim = v->instrs[pr.first + j];
        myrt_sdf_instr const op = v->instrs[pr.first + j + 1];
        float const* q = G + prim.param_offset;
        switch (prim.op) {
          case MYRT_SDF_SPHERE:
            R = std::fabs(double(q[0]));
            bounded = true;
            break;
          case MYRT_SDF_BOX:
            if (q[0] >= 0.f && q[1] >= 0.f && q[2] >= 0.f) {
              R = std::sqrt(double(q[0]) * q[0] + double(q[1]) * q[1] + double(q[2]) * q[2]);
              bounded = true;
            }
            break;
          case MYRT_SDF_TORUS:
            R = std::fabs(double(q[0])) + double(q[1]);
            bounded = true;
            break;
          case MYRT_SDF_CAPSULE:
            if (q[0] >= 0.f) {
              c[1] += 0.5 * double(q[0]);
              R = 0.5 * double(q[0]) + double(q[1]);
              bounded = true;
            }
            break;
          default: break;  // operators, the Menger sponge: no bound
        }
        float k = -1.f;
        if (op.op == MYRT_SDF_UNION) k = 0.f;
        else if (op.op == MYRT_SDF_SMOOTH_UNION && G[op.param_offset] > 0.f) k = G[op.param_offset];
        bool const finite = std::isfinite(R) && std::isfinite(c[0]) && std::isfinite(c[1]) && std::isfinite(c[2]);
        if (k >= 0.f && finite && bounded) {
          // a negative R is a valid (tighter) bound too: distance >= |p - c| - R
          float4 const s = make_float4(float(c[0]), float(c[1]), float(c[2]), float(R) + 1e-6f * float(std::fabs(R)));
          int kbits;
          std::memcpy(&kbits, &k, sizeof kbits);
          int2 const n = make_int2(pr.first + j + 2, kbits);
          if (owner[ag] < 0) {
            owner[ag] = int(p);
            sphere[ag] = s;
            next[ag] = n;
            any = true;
          } else if (next[ag].x != n.x || next[ag].y != n.y || std::memcmp(&sphere[ag], &s, sizeof s) != 0) {
            next[ag] = make_int2(0, 0);  // instruction shared by programs with different groups
          }
        }
      }
      // stack depth after instruction g
      int const op = v->instrs[ag].op;
      if (op >= MYRT_SDF_TRANSLATE) {
      } else if (op >= MYRT_SDF_UNION) {
        --depth;
      } else {
        ++depth;
      }
    }
  }
  if (!any) {
    sphere.clear();
    next.clear();
  }
}

// Per instruction: the number of operator instructions of its program up to and
// including it, so that an evaluation that leaves out a range of instructions
// can still draw the random numbers those operators would have drawn (sdf.cuh
// map, material loads). Empty when programs share instructions at different
// offsets.
inline void sdf_op_counts(myrt_sdf_view const* v, std::vector<int>& out) {
  out.assign(v->instr_count, -1);
  for (size_t p = 0; p < v->program_count; ++p) {
    myrt_sdf_program const pr = v->programs[p];
    int n = 0;
    for (int k = 0; k < pr.count; ++k) {
      int const op = v->instrs[pr.first + k].op;
      if (op >= MYRT_SDF_UNION && op < MYRT_SDF_TRANSLATE) ++n;
      int& slot = out[pr.first + k];
      if (slot >= 0 && slot != n) {
        out.clear();
        return;
      }
      slot = n;
    }
  }
}

// Distance bounds of a primitive about a centre c (updated in place for the
// capsule, whose centre is its segment's midpoint):
//   |p - c| - R  <=  d(p)  <=  |p - c| + U   for every point p.
// Sphere (r): d = |p - c| - r. Box (b >= 0): the box lies within |b| of c and
// holds the ball of radius min(b). Torus (R1, r2): the ring is at |R1| from c.
// Capsule (h >= 0, r): the segment lies within h / 2 of its midpoint.
inline bool sdf_prim_bounds(int op, float const* q, double c[3], double& R, double& U) {
  switch (op) {
    case MYRT_SDF_SPHERE:
      R = std::fabs(double(q[0]));
      U = -double(q[0]);
      return true;
    case MYRT_SDF_BOX:
      if (!(q[0] >= 0.f && q[1] >= 0.f && q[2] >= 0.f)) return false;
      R = std::sqrt(double(q[0]) * q[0] + double(q[1]) * q[1] + double(q[2]) * q[2]);
      U = -double(std::fmin(q[0], std::fmin(q[1], q[2])));
      return true;
    case MYRT_SDF_TORUS:
      R = std::fabs(double(q[0])) + double(q[1]);
      U = std::fabs(double(q[0])) - double(q[1]);
      return true;
    case MYRT_SDF_CAPSULE:
      if (!(q[0] >= 0.f)) return false;
      c[1] += 0.5 * double(q[0]);
      R = 0.5 * double(q[0]) + double(q[1]);
      U = 0.5 * double(q[0]) - double(q[1]);
      return true;
    default: return false;
  }
}

// Per-program cell lists for the evaluator (sdf.cuh map).
//
// Programs that are trees of union / smooth-union operators over translated,
// bounded primitives (any shape: left or right folds, balanced trees) get a
// uniform grid over the primitives' bounding boxes. Two facts about an
// operator op(A, B) with factor k (k = 0 for a union), A the left operand:
//   * it returns A's value bit for bit where B >= A + k (h clamps to 1), and
//     B's where A >= B + k (h clamps to 0), up to the sign of a zero result;
//   * its value lies between min(A, B) - delta and min(A, B): a smooth union
//     never exceeds its smaller operand and falls below it by at most k / 4;
//     when one operand is a primitive it stays above min(lower bounds) -
//     max(delta of the other operand, k) (the blend lowers min(a, b) by
//     (k - |a - b|)^2 / 4k and never below the primitive minus k).
// Every node thus has a lower bound (its primitives' |p - c| - R minus its
// delta) and an upper bound (the smallest |p - c| + U of its primitives) over
// a cell. Walking the tree from the root, an operator whose right subtree's
// lower bound is at least the left's upper bound + k + a rounding margin
// drops the right subtree and itself, and the mirror case drops the left
// subtree and the operator, for every point of the cell. What remains of the
// program is stored as instruction segments in program order; the stack then
// holds the same values as the full evaluation at every step that runs.
// Points outside the grid evaluate the whole program.
//
// Escape sphere: the root's value is at least |p - C| - rho - delta_root with
// rho bounding every primitive's |c_i - C| + R_i, so a march that is outside
// the sphere (C, r_esc) and moving away from C never meets a value below eps
// again (sdf.cuh march).
struct sdf_cells {
  std::vector<int4> hdr;       // 3 per program: (lo.xyz, 1 / cell) bits; (nx, ny, nz, first cell);
                               // escape sphere (C.xyz, r_esc) bits
  std::vector<int> start;      // per program (cells + 1) offsets into list
  std::vector<uint32_t> list;  // segment (start | end << 16), relative to the program's first instruction
  // left folds: a second grid, twice the first one's extent in cells four times
  // as long, whose cells' offsets and segments follow in start and list
  std::vector<int4> outer;     // 2 per program: (lo.xyz, 1 / cell) bits; (nx, ny, nz, first cell), nx = 0: none
};

// As many host threads as there are cores, at most n (and one): n counts pieces of work of a few
// hundred microseconds, since starting 16 threads takes 0.2 ms.
inline int host_threads(size_t n) {
  return int(std::max<size_t>(1, std::min<size_t>(n, std::thread::hardware_concurrency())));
}
template <class F> inline void on_threads(int n, F const& f) {  // f(0) .. f(n - 1)
  std::vector<std::thread> pool;
  for (int t = 1; t < n; ++t) pool.emplace_back(std::cref(f), t);
  f(0);
  for (std::thread& th : pool) th.join();
}

// cells_long: cells along the grid's longest axis (2..128). max_entries: segments that all programs'
// first grids may hold together; the second grids, which only folds have and evaluation can do
// without, hold at most half as many and take nothing from them.
inline void sdf_cell_tables(
    myrt_sdf_view const* v, int cells_long, sdf_cells& out, size_t max_entries = size_t(1) << 26) {
  out = sdf_cells{};
  out.hdr.assign(3 * v->program_count, make_int4(0, 0, 0, 0));
  out.outer.assign(2 * v->program_count, make_int4(0, 0, 0, 0));
  float const* G = v->params;
  struct node {
    int first, end;  // instruction range (end exclusive); an operator's own index is end - 1
    int a = -1, b = -1;  // operand nodes (operators)
    double c[3] = {0.0, 0.0, 0.0}, R = 0.0, U = 0.0;  // primitives
    double k = 0.0, delta = 0.0;
  };
  bool any = false;
  size_t outer_entries = 0;  // of out.list
  for (size_t p = 0; p < v->program_count; ++p) {
    myrt_sdf_program const pr = v->programs[p];
    if (pr.count >= 65536) continue;
    std::vector<node> ns;
    std::vector<int> st;
    int n_prims = 0;
    bool ok = true;
    for (int j = 0; ok && j < pr.count;) {
      myrt_sdf_instr const in = v->instrs[pr.first + j];
      if (in.op == MYRT_SDF_UNION || in.op == MYRT_SDF_SMOOTH_UNION) {
        if (st.size() < 2) { ok = false; break; }
        node n{};
        n.b = st.back();
        st.pop_back();
        n.a = st.back();
        st.pop_back();
        n.first = ns[n.a].first;
        n.end = j + 1;
        if (in.op == MYRT_SDF_SMOOTH_UNION) {
          if (!(G[in.param_offset] > 0.f)) { ok = false; break; }
          n.k = double(G[in.param_offset]);
        }
        bool const leaf_a = ns[n.a].a < 0, leaf_b = ns[n.b].a < 0;
        double const da = ns[n.a].delta, db = ns[n.b].delta;
        // both bounds hold; keep the smaller (two primitives: k / 4; a long
        // fold saturates at k)
        n.delta = std::fmax(da, db) + 0.25 * n.k;
        if (leaf_a || leaf_b) n.delta = std::fmin(n.delta, std::fmax(std::fmax(da, db), n.k));
        st.push_back(int(ns.size()));
        ns.push_back(n);
        ++j;
        continue;
      }
      node n{};
      n.first = j;
      while (j < pr.count && v->instrs[pr.first + j].op == MYRT_SDF_TRANSLATE) {
        float const* t = G + v->instrs[pr.first + j].param_offset;
        for (int a = 0; a < 3; ++a) n.c[a] += double(t[a]);
        ++j;
      }
      if (j >= pr.count) { ok = false; break; }
      myrt_sdf_instr const prim = v->instrs[pr.first + j];
      ok = sdf_prim_bounds(prim.op, G + prim.param_offset, n.c, n.R, n.U) && std::isfinite(n.R) &&
           std::isfinite(n.U) && std::isfinite(n.c[0]) && std::isfinite(n.c[1]) && std::isfinite(n.c[2]);
      ++j;
      n.end = j;
      st.push_back(int(ns.size()));
      ns.push_back(n);
      ++n_prims;
    }
    if (!ok || st.size() != 1 || n_prims < 8) continue;
    int const root = st[0];
    // grid over the primitives' bounding boxes, padded by the largest k
    double lo[3], hi[3], kmax = 0.0, scale = 1.0;
    bool first = true;
    for (node const& n : ns) {
      kmax = std::fmax(kmax, n.k);
      if (n.a >= 0) continue;
      double const r = std::fmax(std::fabs(n.R), std::fabs(n.U));
      for (int a = 0; a < 3; ++a) {
        lo[a] = first ? n.c[a] - r : std::fmin(lo[a], n.c[a] - r);
        hi[a] = first ? n.c[a] + r : std::fmax(hi[a], n.c[a] + r);
        scale = std::fmax(scale, std::fabs(n.c[a]) + r);
      }
      first = false;
    }
    double ext = 0.0;
    for (int a = 0; a < 3; ++a) {
      lo[a] -= kmax + 1e-3;
      hi[a] += kmax + 1e-3;
      ext = std::fmax(ext, hi[a] - lo[a]);
    }
    // host work is cells x nodes: coarser grids for very large programs keep
    // an upload within about 2^26 node bounds (about a second)
    int n_long = cells_long;
    while (n_long > 4 && double(n_long) * n_long * n_long * double(ns.size()) > double(1 << 26)) n_long = n_long * 3 / 4;
    float const inv_f = float(double(n_long) / ext);
    float lo_f[3];
    int dims[3];
    for (int a = 0; a < 3; ++a) {
      lo_f[a] = float(lo[a]);
      dims[a] = std::max(1, std::min(n_long, int(std::ceil((hi[a] - double(lo_f[a])) * double(inv_f)))));
    }
    // Appends the cell lists of one grid to out.start / out.list. False when
    // they would take more than `room` entries.
    // z-slabs of cells on host threads; each keeps its cells' segment counts
    // and segments, concatenated in cell order afterwards
    auto add_grid = [&](float const (&lo_f)[3], float inv_f, int const (&dims)[3], double scale, size_t room) -> bool {
      size_t const ncell = size_t(dims[0]) * dims[1] * dims[2];
      double const cell = 1.0 / double(inv_f);
      // the device finds a point's cell by rounded float arithmetic: widen each
      // cell; the margin covers the rounding of every distance and of the
      // operators' values over the whole program
      double const widen = 1e-4 * cell + 1e-6 * scale;
      double const margin = 2e-3 + 4e-6 * double(n_prims) * scale;
      size_t const first_start = out.start.size();
      size_t const first_entry = out.list.size();
      struct slab {
        std::vector<int> sizes;
        std::vector<uint32_t> segs;
      };
      int const n_threads = host_threads(std::min(size_t(dims[2]), 1 + ncell * ns.size() / (1 << 14)));
      std::vector<slab> slabs(n_threads);
      // the bounds are finite, and std::fmax / std::fmin are calls into the library: 2.5-3 times as long
      auto const max = [](double a, double b) { return a > b ? a : b; };
      auto const min = [](double a, double b) { return a < b ? a : b; };
      auto fill = [&](int t) {
        slab& out_t = slabs[t];
        std::vector<double> lb(ns.size()), ub(ns.size());
        std::vector<int> todo;
        uint32_t seg_s = 0, seg_e = 0;
        bool open = false;
        auto exec = [&](int s0, int e0) {  // append [s0, e0), merging with the open segment
          if (open && int(seg_e) == s0) {
            seg_e = uint32_t(e0);
            return;
          }
          if (open) out_t.segs.push_back(seg_s | (seg_e << 16));
          seg_s = uint32_t(s0);
          seg_e = uint32_t(e0);
          open = true;
        };
        int const z0 = int(int64_t(dims[2]) * t / n_threads), z1 = int(int64_t(dims[2]) * (t + 1) / n_threads);
        for (int z = z0; z < z1; ++z)
          for (int y = 0; y < dims[1]; ++y)
            for (int x = 0; x < dims[0]; ++x) {
              int const idx[3] = {x, y, z};
              double bmin[3], bmax[3];
              for (int a = 0; a < 3; ++a) {
                bmin[a] = double(lo_f[a]) + idx[a] * cell - widen;
                bmax[a] = double(lo_f[a]) + (idx[a] + 1) * cell + widen;
              }
              size_t const before = out_t.segs.size();
              for (size_t i = 0; i < ns.size(); ++i) {  // operands come before their operator
                node const& n = ns[i];
                if (n.a < 0) {
                  double n2 = 0.0, f2 = 0.0;
                  for (int a = 0; a < 3; ++a) {
                    double const o = max(0.0, max(bmin[a] - n.c[a], n.c[a] - bmax[a]));
                    double const f = max(std::fabs(n.c[a] - bmin[a]), std::fabs(n.c[a] - bmax[a]));
                    n2 += o * o;
                    f2 += f * f;
                  }
                  lb[i] = std::sqrt(n2) - n.R;
                  ub[i] = std::sqrt(f2) + n.U;
                } else {
                  // lb of an operator node is (its primitives' smallest bound -
                  // its delta); lb + delta recovers the primitives' bound
                  lb[i] = min(lb[n.a] + ns[n.a].delta, lb[n.b] + ns[n.b].delta) - n.delta;
                  ub[i] = min(ub[n.a], ub[n.b]);
                }
              }
              open = false;
              todo.assign(1, root);
              while (!todo.empty()) {  // depth first, left operand first
                int const i = todo.back();
                todo.pop_back();
                if (i < 0) {  // an operator kept with both operands
                  exec(-i - 1, -i);
                  continue;
                }
                node const& n = ns[i];
                if (n.a < 0) {
                  exec(n.first, n.end);
                  continue;
                }
                if (lb[n.b] >= ub[n.a] + n.k + margin) {
                  todo.push_back(n.a);  // the right operand and the operator drop out
                } else if (lb[n.a] >= ub[n.b] + n.k + margin) {
                  todo.push_back(n.b);  // the left operand and the operator drop out
                } else {
                  todo.push_back(-(n.end - 1) - 1);
                  todo.push_back(n.b);
                  todo.push_back(n.a);
                }
              }
              if (open) out_t.segs.push_back(seg_s | (seg_e << 16));
              out_t.sizes.push_back(int(out_t.segs.size() - before));
            }
      };
      on_threads(n_threads, fill);
      size_t entries = 0;
      for (slab const& sl : slabs) entries += sl.segs.size();
      if (entries > room) return false;
      out.start.reserve(first_start + ncell + 1);
      out.list.reserve(first_entry + entries);
      for (slab const& sl : slabs) {
        for (int n_seg : sl.sizes) {
          out.start.push_back(int(out.list.size()));
          out.list.resize(out.list.size() + size_t(n_seg));
        }
      }
      {  // copy the segments behind the offsets just laid out
        size_t at = first_entry;
        for (slab const& sl : slabs) {
          std::copy(sl.segs.begin(), sl.segs.end(), out.list.begin() + ptrdiff_t(at));
          at += sl.segs.size();
        }
      }
      out.start.push_back(int(out.list.size()));
      return true;
    };
    size_t const first_start = out.start.size();
    size_t const inner = out.list.size() - outer_entries;
    if (!add_grid(lo_f, inv_f, dims, scale, max_entries - inner)) continue;  // too large: no cells for this program
    double const margin = 2e-3 + 4e-6 * double(n_prims) * scale;
    // escape sphere about the grid's centre; the radius carries a relative
    // margin for the rounding of values and positions far from the field
    float esc[4];
    double rho = 0.0;
    for (int a = 0; a < 3; ++a) esc[a] = float(0.5 * (lo[a] + hi[a]));
    for (node const& n : ns) {
      if (n.a >= 0) continue;
      double const dx = n.c[0] - esc[0], dy = n.c[1] - esc[1], dz = n.c[2] - esc[2];
      rho = std::fmax(rho, std::sqrt(dx * dx + dy * dy + dz * dz) + n.R);
    }
    esc[3] = float((rho + ns[root].delta + margin) * 1.001 + 1e-3);
    int lo_bits[3], inv_bits, esc_bits[4];
    std::memcpy(lo_bits, lo_f, sizeof lo_bits);
    std::memcpy(&inv_bits, &inv_f, sizeof inv_bits);
    std::memcpy(esc_bits, esc, sizeof esc_bits);
    out.hdr[3 * p + 0] = make_int4(lo_bits[0], lo_bits[1], lo_bits[2], inv_bits);
    out.hdr[3 * p + 1] = make_int4(dims[0], dims[1], dims[2], int(first_start));
    out.hdr[3 * p + 2] = make_int4(esc_bits[0], esc_bits[1], esc_bits[2], esc_bits[3]);
    any = true;
    bool fold = true;  // every operator's right operand is a primitive
    for (node const& n : ns) fold = fold && (n.a < 0 || ns[n.b].a < 0);
    if (!fold) continue;
    float const inv2 = 0.25f * inv_f;
    float lo2[3];
    int dims2[3];
    double scale2 = scale;
    for (int a = 0; a < 3; ++a) {
      double const half = 0.5 * double(dims[a]) / double(inv_f), mid = double(lo_f[a]) + half;
      lo2[a] = float(mid - 2.0 * half);
      dims2[a] = std::max(1, (2 * dims[a] + 3) / 4);
      scale2 = std::fmax(scale2, std::fabs(mid) + 2.0 * half + 4.0 / double(inv_f));
    }
    size_t const outer_start = out.start.size();
    size_t const before = out.list.size();
    if (!add_grid(lo2, inv2, dims2, scale2, max_entries / 2 - outer_entries)) continue;
    outer_entries += out.list.size() - before;
    int lo2_bits[3], inv2_bits;
    std::memcpy(lo2_bits, lo2, sizeof lo2_bits);
    std::memcpy(&inv2_bits, &inv2, sizeof inv2_bits);
    out.outer[2 * p + 0] = make_int4(lo2_bits[0], lo2_bits[1], lo2_bits[2], inv2_bits);
    out.outer[2 * p + 1] = make_int4(dims2[0], dims2[1], dims2[2], int(outer_start));
  }
  if (!any) out = sdf_cells{};
}

// Compiled left folds. A program that folds bounded primitives from left to
// right -- group 0: [translate] primitive, group g: [translate] primitive,
// union / smooth union -- and has cell lists is also kept as one record per
// group, and each cell's segments as the list of its groups, so that the
// evaluator (sdf.cuh chain_map) runs without decoding instructions and without
// a stack. Record (3 float4): bounding sphere (c, R + k) of the group, as
// sdf_skip_tables; (offset.xyz, kind bits: primitive op | 256 for a union);
// (primitive parameters, k). One more record ends the program's: a sphere of
// radius -inf, skipped at every point, which fills lists up to four entries.
struct sdf_chains {
  std::vector<int4> hdr;        // per program: (first record, groups, full list's first and end batch); groups 0: none
  std::vector<float4> rec;      // 3 per group
  std::vector<int> start;       // parallel to sdf_cells::start: first batch of four entries
  std::vector<uint16_t> list;   // group numbers, lists padded to whole batches with the program's last record
};

inline void sdf_chain_tables(myrt_sdf_view const* v, sdf_cells const& cells, sdf_chains& out) {
  out = sdf_chains{};
  if (cells.list.empty()) return;
  out.hdr.assign(v->program_count, make_int4(0, 0, 0, 0));
  out.start.assign(cells.start.size(), 0);
  float const* G = v->params;
  bool any = false;
  auto bits = [](int i) {
    float f;
    std::memcpy(&f, &i, sizeof f);
    return f;
  };
  for (size_t p = 0; p < v->program_count; ++p) {
    int4 const dims = cells.hdr[3 * p + 1];
    if (dims.x <= 0) continue;
    myrt_sdf_program const pr = v->programs[p];
    std::vector<float4> rec;
    std::vector<int> group(pr.count, -1);    // instruction -> its group
    std::vector<int> group_end;              // group -> the instruction after its last
    std::vector<uint8_t> is_op(pr.count, 0);
    bool ok = true;
    int g = 0;
    for (int j = 0; ok && j < pr.count; ++g) {
      float off[3] = {0.f, 0.f, 0.f};
      myrt_sdf_instr in = v->instrs[pr.first + j];
      if (in.op == MYRT_SDF_TRANSLATE) {  // one translation at most: p - 0 is p, two would round twice
        std::memcpy(off, G + in.param_offset, sizeof off);
        group[j++] = g;
        if (j >= pr.count) { ok = false; break; }
        in = v->instrs[pr.first + j];
      }
      double c[3] = {off[0], off[1], off[2]}, R = 0.0, U = 0.0;
      float const* q = G + in.param_offset;
      if (!sdf_prim_bounds(in.op, q, c, R, U)) { ok = false; break; }
      group[j++] = g;
      int kind = in.op;
      float k = 0.f;
      if (g > 0) {
        if (j >= pr.count) { ok = false; break; }
        myrt_sdf_instr const op = v->instrs[pr.first + j];
        if (op.op == MYRT_SDF_UNION) kind |= 256;
        else if (op.op == MYRT_SDF_SMOOTH_UNION && G[op.param_offset] > 0.f) k = G[op.param_offset];
        else { ok = false; break; }
        is_op[j] = 1;
        group[j++] = g;
      }
      group_end.push_back(j);
      float const Rf = float(R) + 1e-6f * float(std::fabs(R));
      rec.push_back(make_float4(float(c[0]), float(c[1]), float(c[2]), Rf + k));
      rec.push_back(make_float4(off[0], off[1], off[2], bits(kind)));
      bool const box = in.op == MYRT_SDF_BOX;
      rec.push_back(make_float4(q[0], in.op == MYRT_SDF_SPHERE ? 0.f : q[1], box ? q[2] : 0.f, k));
    }
    if (!ok || g < 2 || g >= 65535) continue;
    // the cells' groups (both grids, one after the other), and every group as
    // one more list: counted, then written where they belong, on host threads
    int4 const grid2 = cells.outer[2 * p + 1];
    size_t const n1 = size_t(dims.x) * dims.y * dims.z, n2 = size_t(grid2.x) * grid2.y * grid2.z, ncell = n1 + n2;
    auto cell = [&](size_t i) { return i < n1 ? size_t(dims.w) + i : size_t(grid2.w) + (i - n1); };
    // calls f(first, last) for the groups of each of a cell's segments; false when they are not whole groups
    auto groups = [&](size_t c, auto const& f) {
      int last = -1;
      for (int e = cells.start[c]; e < cells.start[c + 1]; ++e) {
        int j = int(cells.list[e] & 0xffffu);
        int const end = int(cells.list[e] >> 16);
        while (j < end && group[j] == last) ++j;  // the operator of the segment before's last group
        if (j == end) continue;
        // an operator follows its own group's primitive, and a group after the list's first needs its
        // operator in the same segment, as those inside a segment have it
        int const g0 = group[j], g1 = group[end - 1];
        bool const first_op = is_op[std::min(end, group_end[g0]) - 1];
        if (is_op[j] || (last < 0) == first_op || (g1 > g0 && !is_op[end - 1])) return false;
        f(g0, g1);
        last = g1;
      }
      return last >= 0;
    };
    size_t const segments = size_t(cells.start[dims.w + n1] - cells.start[dims.w]);
    int const n_count = host_threads(segments / (1 << 15));
    std::vector<int> batches(ncell);
    std::vector<uint8_t> whole(n_count, 1);
    on_threads(n_count, [&](int t) {
      for (size_t i = ncell * t / n_count; whole[t] && i < ncell * (t + 1) / n_count; ++i) {
        int n = 0;
        whole[t] = groups(cell(i), [&](int g0, int g1) { n += g1 - g0 + 1; });
        batches[i] = (n + 3) / 4;
      }
    });
    size_t entries = 0;
    for (int n : batches) entries += size_t(n);
    for (uint8_t w : whole) ok = ok && w;
    if (!ok || entries + out.list.size() / 4 > (size_t(1) << 28)) continue;
    int at = int(out.list.size() / 4);
    for (size_t i = 0; i < ncell; ++i) {
      out.start[cell(i)] = at;
      at += batches[i];
      if (i + 1 == n1) out.start[dims.w + n1] = at;
    }
    if (n2) out.start[grid2.w + n2] = at;
    int const full = at;
    out.list.resize(4 * (size_t(full) + size_t(g + 3) / 4), uint16_t(g));  // fills lists up
    int const n_fill = host_threads(entries / (1 << 14));
    on_threads(n_fill, [&](int t) {
      for (size_t i = ncell * t / n_fill; i < ncell * (t + 1) / n_fill; ++i) {
        uint16_t* to = out.list.data() + 4 * size_t(out.start[cell(i)]);
        groups(cell(i), [&](int g0, int g1) {
          for (int k = g0; k <= g1; ++k) *to++ = uint16_t(k);
        });
      }
    });
    for (int k = 0; k < g; ++k) out.list[4 * size_t(full) + k] = uint16_t(k);
    out.hdr[p] = make_int4(int(out.rec.size() / 3), g, full, int(out.list.size() / 4));
    rec.push_back(make_float4(0.f, 0.f, 0.f, -HUGE_VALF));
    rec.push_back(make_float4(0.f, 0.f, 0.f, bits(MYRT_SDF_SPHERE)));
    rec.push_back(make_float4(0.f, 0.f, 0.f, 1.f));
    out.rec.insert(out.rec.end(), rec.begin(), rec.end());
    any = true;
  }
  if (!any) out = sdf_chains{};
}

}  // namespace myrt_b200
