// Counts the rays whose wide walk ends without a result (TEST INFRASTRUCTURE ONLY), on scenes whose
// hits lie on one another: usage redo_count CASE LIMIT.  Every result is compared with the binary
// walk's.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "distance_core.cuh"
#include "layout.h"
#include "scene.h"
#include "trace_core.cuh"

static std::mt19937_64 g(11);
static double uniform(double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); }

template <int KIND, class F>
static long walk(const bzr::KindView &K, const std::vector<double> &rays, double tmin, long *bad) {
  std::vector<double> key(64);
  std::vector<uint32_t> ref(64);
  bzr::Stack sk;
  sk.key = key.data();
  sk.ref = ref.data();
  sk.cap = 64;
  sk.stride = 1;
  uint32_t err = 0;
  long redo = 0;
  for (size_t i = 0; i + 6 <= rays.size(); i += 6) {
    const bzr::Ray r = bzr::make_ray(&rays[i], &rays[i + 3], tmin, 1.7976931348623157e308);
    bzr::KState st, want;
    bzr::traverse<KIND, false>(K, r, want, sk, 0, &err, nullptr);
    const F f = bzr::make_ray_f(r, static_cast<const F *>(nullptr));
    if (!f.ok) continue;
    bzr::Trav tv;
    typename F::Bound hl;
    bzr::wtrav_begin<KIND, false>(K, r, f, st, hl, tv, nullptr);
    while (tv.live) {
      bzr::wtrav_to_leaf<KIND, false>(K, r, f, hl, tv, sk, 0, &err, nullptr);
      while (tv.live && tv.post != bzr::kNoLeaf)
        bzr::wtrav_leaf<KIND, false>(K, r, f, st, hl, tv, &err, nullptr);
    }
    if (tv.post == bzr::kRedoLeaf)
      ++redo;
    else
      *bad += std::memcmp(&st.hit, &want.hit, 8) != 0 || st.pos != want.pos;
  }
  *bad += err != 0;
  return redo;
}

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  const std::string name = argv[1];
  bzr::HostScene s;
  int kind = 0;
  double tmin = 0.0;
  std::vector<double> rays;
  auto ray = [&](double ox, double oy, double oz, double dx, double dy, double dz) {
    for (double x : {ox, oy, oz, dx, dy, dz}) rays.push_back(x);
  };
  if (name == "coplanar" || name == "floor") {
    // a flat grid whose every triangle is there three times, its vertices in three orders;
    // "floor": at a power of two from the origins, where distances straddle a high word
    const int m = 24;
    std::vector<double> v;
    std::vector<uint32_t> f;
    const double z = name == "floor" ? -2.0 : -1.7;
    for (int y = 0; y <= m; ++y)
      for (int x = 0; x <= m; ++x) v.insert(v.end(), {x / 3.0 - 4, y / 3.0 - 4, z});
    for (int y = 0; y < m; ++y)
      for (int x = 0; x < m; ++x) {
        const uint32_t a = y * (m + 1) + x, b = a + 1, c = a + m + 1, d = c + 1;
        const uint32_t t[2][3] = {{a, b, c}, {b, d, c}};
        for (auto &q : t)
          for (int k = 0; k < 3; ++k)
            for (int j = 0; j < 3; ++j) f.push_back(q[(j + k) % 3]);
      }
    bzr::add_mesh(s, v.data(), v.size() / 3, f.data(), f.size() / 3);
    for (int i = 0; i < 40000; ++i)
      if (name == "floor")
        ray(uniform(-3, 3), uniform(-3, 3), 0.0, uniform(-1e-9, 1e-9), uniform(-1e-9, 1e-9), -1.0);
      else
        ray(uniform(-3, 3), uniform(-3, 3), 0.0, uniform(-1, 1), uniform(-1, 1), -1.0);
  } else {
    kind = 1;
    std::vector<double> c, r;
    if (name == "shells") {  // concentric spheres a few ulps apart
      for (int i = 0; i < 64; ++i) {
        c.insert(c.end(), {0.25, 0.25, 0.25});
        r.push_back(1.0 + double(int(g() % 17) - 8) * 0x1p-52);
      }
    } else {  // spheres around the origins, a tmin of nearly 0 below it
      tmin = -1e-6;
      for (int i = 0; i < 400; ++i) {
        for (int a = 0; a < 3; ++a) c.push_back(uniform(-3, 3));
        r.push_back(uniform(0.05, 0.3));
      }
    }
    bzr::add_spheres(s, c.data(), r.data(), r.size());
    for (int i = 0; i < 40000; ++i)
      ray(uniform(-4, 4), uniform(-4, 4), uniform(-4, 4), uniform(-1, 1), uniform(-1, 1),
          uniform(-1, 1));
  }
  bzr::Collection &col = s.kind[kind];
  col.present = true;
  col.tree = bzr::build_tree(col.boxes, s.opt);
  const bzr::KindImage im = bzr::flatten(s, kind);
  bzr::KindView v;
  v.present = 1;
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
  v.n_internal = im.n_internal;
  v.n_prims = static_cast<uint32_t>(im.prim_ids.size());
  v.root_ref = im.root_ref;
  v.mixed_ok = im.mixed_ok;
  std::memcpy(v.root_box, im.root_box, sizeof v.root_box);
  long bad = 0;
  const long w = kind == 0 ? walk<0, bzr::RayW>(v, rays, tmin, &bad)
                           : walk<1, bzr::RayW>(v, rays, tmin, &bad);
  const long d = kind == 0 ? walk<0, bzr::RayD>(v, rays, tmin, &bad)
                           : walk<1, bzr::RayD>(v, rays, tmin, &bad);
  std::printf("%s: %ld and %ld of %zu rays ended without a result (FP32, FP64), %ld differ\n",
              name.c_str(), w, d, rays.size() / 6, bad);
  const long limit = std::strtol(argv[2], nullptr, 10);
  return bad || w > limit || d > limit;
}
