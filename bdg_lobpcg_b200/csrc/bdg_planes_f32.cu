// bdg_planes_f32.cu -- the plane passes in FP32.
#include "bdg_planes.cuh"

int bdgd_planes_apply_f32(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                          long long ldy, void *spec, int nc) {
  return planes_apply<float>(c, p, fd, x, ldx, y, ldy, spec, nc);
}
