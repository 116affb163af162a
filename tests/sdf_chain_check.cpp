// Host check of the compiled left folds (myrt_b200/csrc/sdf_skip.hpp
// sdf_chain_tables): evaluates programs in full (every instruction, no
// skipping) and as the device runs a compiled fold (sdf.cuh chain_map: cell or
// outer-cell list, batches of four, bounding spheres, the shared square root),
// with every + and * rounded separately, and sphere-traces rays with and
// without the escape-sphere exits. Prints, per program: groups compiled (0:
// none), points compared, points whose values differ in any bit, points in the
// outer grid, marches compared, hits, marches that differ, marches that began
// inside, groups tested per compiled point.
//
// Usage: sdf_chain_check <dir with instrs.bin programs.bin params.bin> <cells> <rays> <seed>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <iterator>
#include <random>
#include <string>
#include <vector>

#include "../myrt_b200/csrc/sdf_skip.hpp"

using namespace myrt_b200;

namespace {
struct v3 {
  float x, y, z;
};
float gmin(float a, float b) { return b < a ? b : a; }
float gmax(float a, float b) { return a < b ? b : a; }
float gclamp(float v, float lo, float hi) { return gmin(gmax(v, lo), hi); }
float mixf(float a, float b, float t) { return a * (1.f - t) + b * t; }
float len3(v3 v) { return std::sqrt((v.x * v.x + v.y * v.y) + v.z * v.z); }
float len2(float x, float y) { return std::sqrt(x * x + y * y); }

template <class T> std::vector<T> read_all(std::string const& f) {
  std::ifstream s(f, std::ios::binary);
  std::vector<char> b((std::istreambuf_iterator<char>(s)), std::istreambuf_iterator<char>());
  std::vector<T> v(b.size() / sizeof(T));
  std::memcpy(v.data(), b.data(), v.size() * sizeof(T));
  return v;
}

std::vector<myrt_sdf_instr> I;
std::vector<myrt_sdf_program> P;
std::vector<float> G;
sdf_cells C;
sdf_chains H;
long tested = 0, in_outer = 0;

float full_map(int prog, v3 p) {
  myrt_sdf_program const pr = P[prog];
  std::vector<float> st;
  v3 pos = p;
  for (int k = 0; k < pr.count; ++k) {
    myrt_sdf_instr const in = I[pr.first + k];
    float const* q = G.data() + in.param_offset;
    float d;
    switch (in.op) {
      case MYRT_SDF_TRANSLATE: pos = v3{pos.x - q[0], pos.y - q[1], pos.z - q[2]}; continue;
      case MYRT_SDF_SPHERE: d = len3(pos) - q[0]; break;
      case MYRT_SDF_BOX: {
        v3 const w{std::fabs(pos.x) - q[0], std::fabs(pos.y) - q[1], std::fabs(pos.z) - q[2]};
        d = len3(v3{gmax(w.x, 0.f), gmax(w.y, 0.f), gmax(w.z, 0.f)}) + gmin(gmax(w.x, gmax(w.y, w.z)), 0.f);
        break;
      }
      case MYRT_SDF_TORUS: d = len2(len2(pos.x, pos.z) - q[0], pos.y) - q[1]; break;
      case MYRT_SDF_CAPSULE: {
        v3 w = pos;
        w.y -= gclamp(w.y, 0.f, q[0]);
        d = len3(w) - q[1];
        break;
      }
      default: {
        float const d1 = st.back();
        st.pop_back();
        float const d0 = st.back();
        st.pop_back();
        if (in.op == MYRT_SDF_UNION) {
          d = gmin(d0, d1);
        } else if (in.op == MYRT_SDF_SUBTRACTION) {
          d = gmax(-d0, d1);
        } else {
          float const k2 = q[0];
          float const h = gclamp(0.5f + 0.5f * (d1 - d0) / k2, 0.f, 1.f);
          d = mixf(d1, d0, h) - k2 * h * (1.f - h);
        }
      }
    }
    st.push_back(d);
    pos = p;
  }
  return st.back();
}

bool grid_cell(int4 g0, int4 g1, v3 p, int& c) {
  float lo[3], inv;
  std::memcpy(lo, &g0, sizeof lo);
  std::memcpy(&inv, &g0.w, sizeof inv);
  float const fx = (p.x - lo[0]) * inv, fy = (p.y - lo[1]) * inv, fz = (p.z - lo[2]) * inv;
  if (!(fx >= 0.f && fy >= 0.f && fz >= 0.f && fx < float(g1.x) && fy < float(g1.y) && fz < float(g1.z))) return false;
  c = g1.w + (int(fz) * g1.y + int(fy)) * g1.x + int(fx);
  return true;
}

float chain_map(int prog, v3 p) {
  int4 const ch = H.hdr[prog];
  float const margin = 1e-4f + 1e-6f * ((std::fabs(p.x) + std::fabs(p.y)) + std::fabs(p.z));
  int b = ch.z, e = ch.w, c;
  bool const inner = grid_cell(C.hdr[3 * prog], C.hdr[3 * prog + 1], p, c);
  if (inner || grid_cell(C.outer[2 * prog], C.outer[2 * prog + 1], p, c)) {
    b = H.start[c];
    e = H.start[c + 1];
    in_outer += !inner;
  }
  float4 const* rec = H.rec.data() + 3 * size_t(ch.x);
  float d = 3.402823466e+38f;
  bool first = true;
  for (; b < e; ++b) {
    uint32_t keep = 0;
    float q2[4], w[4];
    for (int h = 0; h < 4; ++h) {
      float4 const sp = rec[3 * H.list[4 * size_t(b) + h]];
      float const qx = p.x - sp.x, qy = p.y - sp.y, qz = p.z - sp.z;
      q2[h] = std::fma(qz, qz, std::fma(qy, qy, qx * qx));
      w[h] = sp.w + margin;
      float const thr = d + w[h];
      if (thr > 0.f && !(q2[h] >= thr * thr)) keep |= 1u << h;
      ++tested;
    }
    for (int h = 0; h < 4; ++h) {
      if (!(keep >> h & 1u)) continue;
      float const thr = d + w[h];
      if (!(thr > 0.f) || q2[h] >= thr * thr) continue;
      size_t const g = H.list[4 * size_t(b) + h];
      float4 const a = rec[3 * g + 1], q = rec[3 * g + 2];
      int kind;
      std::memcpy(&kind, &a.w, sizeof kind);
      v3 pos{p.x - a.x, p.y - a.y, p.z - a.z};
      float out = q.x;
      switch (kind & 255) {
        case MYRT_SDF_SPHERE: break;
        case MYRT_SDF_BOX: {
          v3 const x{std::fabs(pos.x) - q.x, std::fabs(pos.y) - q.y, std::fabs(pos.z) - q.z};
          pos = v3{gmax(x.x, 0.f), gmax(x.y, 0.f), gmax(x.z, 0.f)};
          out = -gmin(gmax(x.x, gmax(x.y, x.z)), 0.f);
          break;
        }
        case MYRT_SDF_TORUS:
          pos = v3{len2(pos.x, pos.z) - q.x, pos.y, 0.f};
          out = q.y;
          break;
        default:
          pos.y -= gclamp(pos.y, 0.f, q.x);
          out = q.y;
      }
      float const d1 = len3(pos) - out;
      if (first) {
        d = d1;
        first = false;
      } else if (!(d1 - d >= q.w)) {
        if (kind & 256) {
          d = gmin(d, d1);
        } else {
          float const t = gclamp(0.5f + 0.5f * (d1 - d) / q.w, 0.f, 1.f);
          d = mixf(d1, d, t) - q.w * t * (1.f - t);
        }
      }
    }
  }
  return d;
}

bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0 || (a == 0.f && b == 0.f) || (a != a && b != b); }

// raymarch.glsl:116-145; fast: compiled evaluation and the escape exits
bool march(int prog, v3 ro, v3 rd, bool fast, int& si, float& t_hit, std::vector<v3>* pts) {
  float const eps = 1e-4f;
  float const len = len3(rd);
  float t = 10.f * eps;
  si = 0;
  float e[4];
  std::memcpy(e, &C.hdr[3 * prog + 2], sizeof e);
  float const er = e[3] + eps;
  for (int i = 0; i < 256 && t / len < __builtin_huge_valf(); ++i) {
    v3 const q{ro.x + rd.x * t / len, ro.y + rd.y * t / len, ro.z + rd.z * t / len};
    float const m = fast ? chain_map(prog, q) : full_map(prog, q);
    if (pts) pts->push_back(q);
    if (si == 0) si = m > 0.f ? 1 : (m < 0.f ? -1 : 0);
    if (std::fabs(m) < eps) {
      t_hit = t;
      return t >= 0.f;
    }
    if (fast) {
      v3 const w{q.x - e[0], q.y - e[1], q.z - e[2]};
      float const away = (w.x * rd.x + w.y * rd.y) + w.z * rd.z;
      if ((si > 0 ? away >= 0.f : (si < 0 && m > 0.f && away <= 0.f)) &&
          (w.x * w.x + w.y * w.y) + w.z * w.z >= er * er)
        return false;
    }
    t += float(si) * m;
  }
  return false;
}
}  // namespace

int main(int argc, char** argv) {
  if (argc < 5) return 2;
  std::string const dir = argv[1];
  I = read_all<myrt_sdf_instr>(dir + "/instrs.bin");
  P = read_all<myrt_sdf_program>(dir + "/programs.bin");
  G = read_all<float>(dir + "/params.bin");
  myrt_sdf_view v{};
  v.instrs = I.data(), v.instr_count = I.size();
  v.programs = P.data(), v.program_count = P.size();
  v.params = G.data(), v.param_count = G.size();
  sdf_cell_tables(&v, std::atoi(argv[2]), C);
  sdf_chain_tables(&v, C, H);
  int const n_rays = std::atoi(argv[3]);
  std::mt19937 rng(unsigned(std::atoi(argv[4])));
  std::uniform_real_distribution<float> U(-1.f, 1.f);
  for (size_t p = 0; p < P.size(); ++p) {
    int const groups = H.hdr.empty() ? 0 : H.hdr[p].y;
    long points = 0, bad = 0, marches = 0, hits = 0, bad_marches = 0, inside = 0;
    tested = in_outer = 0;
    for (int n = 0; groups > 0 && n < n_rays; ++n) {
      float const spread = n % 3 == 0 ? 0.7f : (n % 3 == 1 ? 2.f : 6.f);
      v3 ro{U(rng) * spread, U(rng) * spread, U(rng) * spread};
      v3 rd{U(rng), U(rng), U(rng)};
      if (n % 5 == 0) rd = v3{-ro.x + U(rng), -ro.y + U(rng), -ro.z + U(rng)};  // toward the field
      if (n % 7 == 0) rd = v3{0.f, rd.y < 0.f ? -1.f : 1.f, 0.f};
      float const l = len3(rd);
      if (!(l > 1e-3f)) continue;
      rd = v3{rd.x / l, rd.y / l, rd.z / l};
      std::vector<v3> pts;
      int s0, s1;
      float t0 = 0.f, t1 = 0.f;
      bool const h0 = march(int(p), ro, rd, false, s0, t0, &pts);
      bool const h1 = march(int(p), ro, rd, true, s1, t1, nullptr);
      ++marches;
      hits += h0;
      inside += s0 < 0;
      bad_marches += h0 != h1 || (h0 && !same(t0, t1)) || s0 != s1;
      for (size_t k = 0; k < pts.size() && k < 40; ++k) {
        ++points;
        bad += !same(full_map(int(p), pts[k]), chain_map(int(p), pts[k]));
      }
    }
    std::printf("%d %ld %ld %ld %ld %ld %ld %ld %.1f\n", groups, points, bad, in_outer, marches, hits, bad_marches,
        inside, points ? double(tested) / double(points) : 0.0);
  }
  return 0;
}
