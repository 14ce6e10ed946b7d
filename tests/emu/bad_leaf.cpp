// A leaf reference past the arrays (TEST INFRASTRUCTURE ONLY; built with AddressSanitizer): both
// wide walks, counting and not, flag it and read nothing there.
#include <cstdio>
#include <cstring>
#include <vector>

#include "distance_core.cuh"
#include "layout.h"
#include "scene.h"
#include "trace_core.cuh"

template <bool COUNT, class F>
static bool flagged(const bzr::KindView &K, const bzr::Ray &r) {
  std::vector<double> key(64);
  std::vector<uint32_t> ref(64);
  bzr::Stack sk;
  sk.key = key.data();
  sk.ref = ref.data();
  sk.cap = 64;
  sk.stride = 1;
  bzr::KState st;
  bzr::Counts c = {};
  uint32_t err = 0;
  bzr::traverse_mixed<bzr::kSpheres, COUNT, F>(K, r, st, sk, 0, &err, &c);
  return (err & bzr::kErrPrimIndex) != 0;
}

int main() {
  bzr::HostScene s;
  std::vector<double> c, rad;
  for (int i = 0; i < 60; ++i) {
    for (int a = 0; a < 3; ++a) c.push_back(a == 0 ? 0.5 * i : 0.0);
    rad.push_back(0.2);
  }
  bzr::add_spheres(s, c.data(), rad.data(), rad.size());
  bzr::Collection &col = s.kind[bzr::kSpheres];
  col.present = true;
  col.tree = bzr::build_tree(col.boxes, s.opt);
  bzr::KindImage im = bzr::flatten(s, bzr::kSpheres, 1, false);
  const uint32_t n = static_cast<uint32_t>(im.prim_ids.size());
  std::vector<double> box(6 * size_t(n), 0.0);
  bzr::KindView v;
  v.present = 1;
  v.nodes64 = im.nodes64.data();
  v.wide = im.wide.data();
  v.leaf_box = box.data();
  v.n_wide = im.n_wide;
  v.wide_root_ref = im.wide_root_ref;
  v.payload = im.payload.data();
  v.prim_ids = im.prim_ids.data();
  v.n_internal = im.n_internal;
  v.n_prims = n;
  v.root_ref = im.root_ref;
  v.mixed_ok = im.mixed_ok;
  std::memcpy(v.root_box, im.root_box, sizeof v.root_box);
  if (!im.mixed_ok || (im.wide_root_ref & bzr::kLeafBit)) return 2;
  // every leaf of the image past the arrays
  for (uint32_t g = 0; g < im.n_wide; ++g) {
    uint32_t refs[8];
    unsigned char *nd = &im.wide[size_t(g) * bzr::kWideBytes];
    std::memcpy(refs, nd + 64, sizeof refs);
    for (uint32_t &x : refs)
      if (x & bzr::kLeafBit) x = bzr::kLeafBit | (n + 1000);
    std::memcpy(nd + 64, refs, sizeof refs);
  }
  const double o[3] = {-5, 0.01, 0.02}, d[3] = {1, 1e-3, 1e-3};
  const bzr::Ray r = bzr::make_ray(o, d, 0.0, 1.7976931348623157e308);
  const bool all = flagged<false, bzr::RayW>(v, r) && flagged<false, bzr::RayD>(v, r) &&
                   flagged<true, bzr::RayW>(v, r) && flagged<true, bzr::RayD>(v, r);
  std::printf("flagged: %d\n", all);
  return all ? 0 : 1;
}
