// bdg_planes.h -- 3D operator applies in three passes: a whole xy plane per
// block forward, z lines, a whole xy plane per block inverse
// (bdg_planes.cuh).  Internal to the library.
#pragma once

#include "bdg_dev.h"
#include "bdg_kern.cuh"

// Whether the plane kernels can run an apply on context c: a 3D grid whose
// axes split into two factors of at most 16 and whose plane of one spectrum
// fits one block's shared memory.
bool bdgd_planes_usable(const bdgd_ctx *c, int prec);

// Whether an apply of few columns is better done by plane passes than by line
// passes, on a context where both can run.
bool bdgd_planes_pay(const bdgd_ctx *c, const Prog &p, int prec, int nc);

// Full operator apply of program p on nc columns; spec holds nc * p.J spectra.
int bdgd_planes_apply_f64(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                          long long ldy, void *spec, int nc);
int bdgd_planes_apply_f32(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                          long long ldy, void *spec, int nc);
