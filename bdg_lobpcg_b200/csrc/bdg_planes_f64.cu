// bdg_planes_f64.cu -- the plane passes in FP64 and their geometry.
#include "bdg_planes.cuh"

static FDiv make_fdiv(int d) {
  FDiv f;
  f.d = (unsigned)d;
  f.m = (unsigned)((0x100000000ull + (unsigned)d - 1) / (unsigned)d);
  return f;
}

// n = a * b with 2 <= a <= b <= 16 and b - a smallest; false if there is none
static bool split2(int n, int *a, int *b) {
  *a = split_small(n);
  if (!*a) return false;
  *b = n / *a;
  return true;
}

bool bdgd_plane_par(const bdgd_ctx *c, PlaneGeo *q) {
  if (c->dim != 3) return false;
  q->nx = c->N[0];
  q->ny = c->N[1];
  q->nz = c->N[2];
  q->nxk = c->nxk;
  int a, b;
  if (!split2(q->nx, &q->x1, &q->x2)) return false;
  if (!split2(q->ny, &a, &b)) return false;
  q->mode = c->cplx ? PL_CPLX : q->ny % 2 == 0 ? PL_REAL : PL_WHOLE;
  q->ye = q->mode == PL_REAL && a % 2 ? b : a;
  q->yo = q->ny / q->ye;
  if (!split2(q->nz, &q->z2, &q->z1)) return false;
  q->rows = q->mode == PL_REAL ? q->ny / 2 : q->ny;
  q->x2p = q->x2 | 1;
  q->ex = q->x1 * q->x2p;
  q->ld = q->ex + (q->mode == PL_REAL ? 2 : 0);
  const int ldm = q->x2 % 8 ? q->x2 % 8 : q->x1 % 8;  // see PlaneCT::ld
  while (q->ld % 8 != ldm) q->ld++;
  q->dx1 = make_fdiv(q->x1);
  q->dx2 = make_fdiv(q->x2);
  q->dnxk = make_fdiv(q->nxk);
  q->dyr = make_fdiv(q->mode == PL_REAL ? q->ye / 2 : q->ye);
  q->tx = 16;
  return true;
}

bool bdgd_planes_usable(const bdgd_ctx *c, int prec) {
  PlaneGeo q;
  if (!bdgd_plane_par(c, &q)) return false;
  const size_t csz = prec == BDGD_F32 ? sizeof(float2) : sizeof(double2);
  return csz * (size_t)q.rows * q.ld <= 227 * 1024;
}

int bdgd_planes_apply_f64(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                          long long ldy, void *spec, int nc) {
  return planes_apply<double>(c, p, fd, x, ldx, y, ldy, spec, nc);
}
