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

// Few columns leave the plane kernels a handful of blocks: a plane is then one
// block's serial work and the kernel takes as long as one block, where the line
// passes still spread over the SMs and cost their launches and bytes.  So the
// plane kernels' time is measured by the rounds of blocks (of all plane kernels)
// times the items a thread works through, that of the line passes by a constant
// for their five launches and the MB of the spectra (axes of 48 and 96 points, whose
// line plans use fewer lanes, at half as much again each), and the planes are
// taken while their share stays below a line; M alone, one half with two
// fields, has a second inverse launch and so a lower one.  Not by that model: the
// cubes with compiled-in sizes always pay (M 128^3 FP64, one column: 73 against
// 102 us), FP32 complex planes that fill an SM do not (T 128^3: 159 against 103),
// nor x = 256 with local terms, nor M with z = 256.
//
// Fitted to one to three columns of K, M, Lrep and T on 40 grids of 16 to 256
// points an axis, real and complex, both precisions (768 cases, microseconds a
// call): always planes is 5.8% behind the better of the two on average (worst
// 2.15x: 128x128x16 complex FP32 M, 64 against 30 us), always lines 17%, this
// rule 1.3% (worst 1.35x).
bool bdgd_planes_pay(const bdgd_ctx *c, const Prog &p, int prec, int nc) {
  PlaneGeo q;
  if (!bdgd_plane_par(c, &q)) return false;
  if (q.mode == PL_REAL && q.nx == q.ny && q.ny == q.nz &&
      (q.nx == 16 || q.nx == 32 || q.nx == 48 || q.nx == 64 || q.nx == 96 || q.nx == 128))
    return true;
  const bool f32 = prec == BDGD_F32;
  const size_t csz = f32 ? sizeof(float2) : sizeof(double2), sm = csz * (size_t)q.rows * q.ld;
  const bool two = p.nf[0] > 1 || (p.nh > 1 && p.nf[1] > 1);
  const bool m_alone = p.nh == 1 && two;
  if (q.mode == PL_CPLX && f32 && 2 * (sm + 1024) > 227 * 1024 && p.J > 1) return false;
  if (q.nx == 256 && (two || p.nh == 1)) return false;
  if (q.nz == 256 && m_alone) return false;
  const bool big = q.x2 > 8 || q.ye > 8 || q.yo > 8;
  int res = f32 ? (big ? 2 : 4) : (big ? 2 : 3);  // blocks an SM, as in plane_blocks()
  const int fit = (int)((size_t)(228 * 1024) / (sm + 1024));
  if (fit < res) res = fit < 1 ? 1 : fit;
  const int slots = 148 * res;
  auto rounds = [&](int blocks) { return (blocks + slots - 1) / slots; };
  const double w = rounds(p.J * nc * q.nz) + rounds(p.nh * nc * q.nz) + (two ? rounds(nc * q.nz) : 0);
  const double items = (double)q.rows * (q.x1 > q.x2 ? q.x1 : q.x2) / 256;
  const double mb = 1e-6 * (double)csz * nc * p.J * c->geo.H;
  const int thirds = (q.nx % 3 == 0) + (q.ny % 3 == 0) + (q.nz % 3 == 0);
  return w * (items + 0.3) <= (m_alone ? 0.22 : 0.34) * (20.0 + mb * (1.0 + 0.5 * thirds));
}

int bdgd_planes_apply_f64(bdgd_ctx *c, const Prog &p, const FieldsDev &fd, const void *x, long long ldx, void *y,
                          long long ldy, void *spec, int nc) {
  return planes_apply<double>(c, p, fd, x, ldx, y, ldy, spec, nc);
}
