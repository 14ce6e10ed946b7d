// Walks the wide image with leaf records (TEST INFRASTRUCTURE ONLY): a view filled from flatten's
// default image by hand, both wide walks against the binary one.  usage: records_walk KIND PRIMS
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "distance_core.cuh"
#include "layout.h"
#include "scene.h"
#include "trace_core.cuh"

static std::mt19937_64 g(7);
static double uniform(double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); }

template <int KIND>
static int run(const bzr::KindView &K, uint32_t cap) {
  std::vector<double> key(cap);
  std::vector<uint32_t> ref(cap);
  bzr::Stack sk;
  sk.key = key.data();
  sk.ref = ref.data();
  sk.cap = cap;
  sk.stride = 1;
  int bad = 0, hits = 0;
  uint32_t err = 0;
  for (int i = 0; i < 20000; ++i) {
    double o[3], d[3];
    for (int a = 0; a < 3; ++a) o[a] = uniform(-3, 3), d[a] = uniform(-1, 1);
    const bzr::Ray r = bzr::make_ray(o, d, 0.0, 1.7976931348623157e308);
    bzr::KState st[3];
    bool h[3];
    h[0] = bzr::traverse<KIND, false>(K, r, st[0], sk, 0, &err, nullptr);
    h[1] = bzr::traverse_mixed<KIND, false>(K, r, st[1], sk, 0, &err, nullptr);
    h[2] = bzr::traverse_mixed<KIND, false, bzr::RayD>(K, r, st[2], sk, 0, &err, nullptr);
    hits += h[0];
    for (int j = 1; j < 3; ++j)
      bad += h[j] != h[0] || std::memcmp(&st[j].hit, &st[0].hit, 8) || st[j].pos != st[0].pos;
  }
  std::printf("%d hits, %d differ, error word %u\n", hits, bad, err);
  return bad || err || hits == 0;
}

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  const char *names[3] = {"mesh", "spheres", "planes"};
  int kind = 0;
  while (kind < 3 && std::strcmp(names[kind], argv[1])) ++kind;
  const size_t n = std::strtoull(argv[2], nullptr, 10);
  if (kind == 3 || n == 0) return 2;
  bzr::HostScene s;
  std::vector<double> c, r, rot;
  for (size_t i = 0; i < n; ++i) {
    for (int a = 0; a < 3; ++a) c.push_back(n == 1 ? 0.0 : uniform(-2, 2));
    r.push_back(n == 1 ? 1.5 : uniform(0.05, 0.3));
    for (int a = 0; a < 9; ++a) rot.push_back(a % 4 == 0 ? 1.0 : 0.0);
  }
  if (kind == 0) {
    std::vector<double> v;
    std::vector<uint32_t> f;
    for (size_t i = 0; i < n; ++i)
      for (int j = 0; j < 3; ++j) {
        for (int a = 0; a < 3; ++a) v.push_back(c[3 * i + a] + uniform(-1.0, 1.0) * r[i] * 2);
        f.push_back(static_cast<uint32_t>(3 * i + j));
      }
    bzr::add_mesh(s, v.data(), v.size() / 3, f.data(), n);
  } else if (kind == 1) {
    bzr::add_spheres(s, c.data(), r.data(), n);
  } else {
    bzr::add_planes(s, c.data(), r.data(), r.data(), rot.data(), n);
  }
  bzr::Collection &col = s.kind[kind];
  col.present = true;
  col.geom_id = 0;
  col.tree = bzr::build_tree(col.boxes, s.opt);
  const bzr::KindImage im = bzr::flatten(s, kind);
  bzr::KindView v;
  v.present = 1;
  v.geom_id = 0;
  v.nodes64 = im.nodes64.data();
  v.wide = im.wide.data();
  v.leaves = im.leaves.data();
  v.n_wide = im.n_wide;
  v.n_leaf16 = im.n_leaf16;
  v.wide_root_ref = im.wide_root_ref;
  v.payload = im.payload.data();
  v.prim_ids = im.prim_ids.data();
  v.tri = im.tri.data();
  v.verts = im.verts.data();
  v.vnorm = im.vnorm.data();
  v.n_internal = im.n_internal;
  v.n_prims = static_cast<uint32_t>(im.prim_ids.size());
  v.n_verts = static_cast<uint32_t>(im.verts.size() / bzr::kVertexDoubles);
  v.root_ref = im.root_ref;
  v.mixed_ok = im.mixed_ok;
  std::memcpy(v.root_box, im.root_box, sizeof v.root_box);
  v.coord_max = im.coord_max;
  if (!im.mixed_ok) {
    std::printf("no wide image\n");
    return 1;
  }
  const uint32_t cap = 64;
  return kind == 0 ? run<0>(v, cap) : kind == 1 ? run<1>(v, cap) : run<2>(v, cap);
}
