// Prints the box of boundary nodes and the frame's descriptors that the kernels get
// for an 8 x 6 lattice: without a mask, without one but with a frame, with a mask
// and no frame, with both.
#include <cstdio>
#include <cstring>

#include "lbm_fused.cuh"

int main() {
  static const uint32_t word = 0;  // never read here
  for (int k = 0; k < 4; ++k) {
    lbm_geometry g;
    std::memset(&g, 0, sizeof(g));
    g.nx = 8;
    g.ny = 6;
    if (k >= 2) g.bcmask = g.desc = &word;
    if (k % 2) {
      g.frame = 1;
      for (int i = 0; i < 8; ++i) g.frame_desc[i] = 1u + i;
      const int box[4] = {2, 4, 1, 3};
      std::memcpy(g.inner_box, box, sizeof(box));
    }
    lbm::GeoK q;
    std::memset(&q, 0, sizeof(q));
    if (!lbm::to_geok(&g, q)) return 1;
    std::printf("%d %d %d %d %u %u\n", q.box_x0, q.box_x1, q.box_y0, q.box_y1, q.frame_desc[0], q.frame_desc[7]);
  }
  return 0;
}
