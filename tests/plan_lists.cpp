// Prints the work lists that build_plan makes for one chain call, for
// test_flag_lists.py. Arguments: width height ssx ssy planes extra columns and
// rows of the input planes, loop-restoration columns and unit size, and which
// of the planes' loop-filter levels are set (a mask).
#include <cstdio>
#include <cstdlib>

#include "plan.h"

using namespace av1pf;

int main(int argc, char** argv) {
  if (argc != 11) return 2;
  int a[10];
  for (int k = 0; k < 10; k++) a[k] = std::atoi(argv[k + 1]);
  const int w = a[0], h = a[1], ssx = a[2], ssy = a[3], np = a[4], mask = a[9];
  av1pf_frame_info i{};
  i.bit_depth = 10;
  i.sample_bytes = 2;
  i.subsampling_x = ssx;
  i.subsampling_y = ssy;
  i.num_planes = np;
  i.frame_width = i.upscaled_width = w;
  i.frame_height = h;
  i.mi_cols = 2 * ((w + 7) >> 3);
  i.mi_rows = 2 * ((h + 7) >> 3);
  av1pf_params p{};
  p.loop_filter_level[0] = p.loop_filter_level[1] = mask & 1 ? 20 : 0;
  p.loop_filter_level[2] = mask & 2 ? 20 : 0;
  p.loop_filter_level[3] = mask & 4 ? 20 : 0;
  p.cdef_enabled = 1;
  p.cdef_damping = 3;
  p.uses_lr = 1;
  av1pf_plane in[3]{}, out[3]{};
  for (int k = 0; k < np; k++) {
    const int sx = k ? ssx : 0, sy = k ? ssy : 0, us = a[8];
    p.frame_restoration_type[k] = 3;
    p.loop_restoration_size[k] = us;
    p.lr_unit_rows[k] = (((h + sy) >> sy) + us / 2) / us > 1 ? (((h + sy) >> sy) + us / 2) / us : 1;
    p.lr_unit_cols[k] = (((w + sx) >> sx) + us / 2) / us > 1 ? (((w + sx) >> sx) + us / 2) / us : 1;
    in[k].data = reinterpret_cast<void*>(4096);
    in[k].width = ((i.mi_cols * 4) >> sx) + 8 + a[5];
    in[k].height = ((i.mi_rows * 4) >> sy) + 8 + a[6];
    in[k].stride = (in[k].width + 63) / 64 * 64;
    out[k] = in[k];
  }
  std::string why;
  if (validate_frame(&i, &p, in, &why) != AV1PF_OK) return std::fprintf(stderr, "%s\n", why.c_str()), 1;
  av1pf_maps m{};
  FrameJob j{&i, &p, &m, in, nullptr, out, reinterpret_cast<uint8_t*>(4096), ST_CHAIN, false};
  j.lf_mode = 3;
  j.lr_cols = a[7];
  Plan plan;
  if (build_plan(&j, 1, nullptr, plan, &why) != AV1PF_OK) return std::fprintf(stderr, "%s\n", why.c_str()), 1;
  const FrameDesc& d = plan.frames[0];
  std::printf("frame %d %zu %d %d %d\n", plan.flag_sync, plan.n_flags, plan.cdef.half, d.cdef_flag_base, d.cdef_sbc);
  for (int k = 0; k < np; k++) std::printf("plane %d %d %d\n", k, d.lf_flag_base[k], d.lf_tiles_x[k]);
  auto list = [](const char* name, const std::vector<Item>& v) {
    for (const Item& it : v)
      std::printf("%s %d %d %d %d %d %d %d %d\n", name, it.plane, it.kind, it.x0, it.y0, it.x1, it.y1, it.a, it.b);
  };
  list("lf", plan.lff_items);
  list("cdef", plan.cdef_items);
  list("lr", plan.lr_items);
  return 0;
}
