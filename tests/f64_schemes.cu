// The guarded fast fluxes of the FP64 schemes (fv_f64.cuh, fv_schemes.cuh) against
// their plain expressions on single faces, at operands around every guard.  For
// each scheme and kind of operands prints the faces the guard lets pass and those
// of them whose fluxes differ from the plain ones (as numbers: a zero's sign may
// differ; NaN equals NaN); exits 1 when any does.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "fv_schemes.cuh"

struct Face {
  double cell[4][5];   // c-2, c-1 | c, c+1
  double A;
  int dir, sl, sr;
};

template <class Scheme>
__global__ void compare(const Face* faces, int n, int* passed, int* wrong, int* first)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const Face& f = faces[t];
  dn::FaceCells c;
  c.sl = f.sl;
  c.sr = f.sr;
  c.s2 = 1;
  c.m1 = f.cell[1];
  c.p0 = f.cell[2];
  c.m2 = f.sl ? f.cell[0] : c.m1;
  c.p1 = f.sr ? f.cell[3] : c.p0;
  dn::Guard g;
  double vl[5], vr[5], F[5], P[5];
  dn::limited_states<1>(c, vl, vr, g);
  Scheme::fast(f.dir, vl, vr, f.A, F, g);
  if (g.any()) return;
  atomicAdd(passed, 1);
  dn::face_flux_plain<Scheme, 1>(f.dir, c, f.A, P);
  bool same = true;
  for (int v = 0; v < 5; ++v) same = same && (F[v] == P[v] || (F[v] != F[v] && P[v] != P[v]));
  if (!same) {
    atomicAdd(wrong, 1);
    atomicMin(first, t);
  }
}

static std::mt19937_64 rng(11);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int pick(int n) { return (int)(rng() % n); }

static double ones(double x)   // upper 19 or 20 significand bits of ones
{
  unsigned long long u;
  std::memcpy(&u, &x, 8);
  u |= pick(2) ? 0x000fffff00000000ull : 0x000ffffe00000000ull;
  std::memcpy(&x, &u, 8);
  return x;
}

static const char* kKinds[] = {"flow", "equal", "tiny", "ones", "sonic", "small", "large", "edges", "invalid"};

static Face face(int kind)
{
  Face f;
  f.dir = pick(3);
  f.sl = pick(4) != 0;
  f.sr = pick(4) != 0;
  f.A = kind == 7 && pick(3) == 0 ? std::ldexp(uni(1, 2), pick(2) ? -310 : 299) : std::exp(uni(-9, 0));
  const double r0 = uni(0.5, 2), T0 = uni(200, 400), a = std::sqrt(dn::Gas::gamma * dn::Gas::R * T0);
  double u0[3];
  for (double& u : u0) u = uni(-2, 2) * a;
  for (int c = 0; c < 4; ++c) {
    const double amp = kind == 1 && pick(3) ? 0 : std::exp2(uni(-40, -2));
    const double r = r0 * (1 + amp * uni(-1, 1)), T = T0 * (1 + amp * uni(-1, 1));
    double u[3];
    for (int d = 0; d < 3; ++d) u[d] = u0[d] * (1 + amp * uni(-1, 1));
    if (kind == 2)
      for (double& x : u) x = pick(4) ? std::ldexp(uni(-1, 1), -pick(1075)) : (pick(2) ? 0.0 : -0.0);
    if (kind == 4) u[f.dir] = std::sqrt(dn::Gas::gamma * dn::Gas::R * T) * (pick(2) ? 1 : -1) * (1 + (pick(5) - 2) * std::ldexp(1.0, -52));
    f.cell[c][0] = r;
    for (int d = 0; d < 3; ++d) f.cell[c][1 + d] = r * u[d];
    f.cell[c][4] = r * (dn::Gas::cv * T + 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]));
    for (int v = 0; v < 5; ++v) {
      double& x = f.cell[c][v];
      if (kind == 3 && pick(3) == 0) x = ones(x);
      if (kind == 5) x = std::ldexp(x, -(280 + pick(60)));
      if (kind == 6) x = std::ldexp(x, 220 + pick(90));
      // differences at the limiter's 1e-10, the ends of the guarded ranges
      if (kind == 7 && c && pick(3) == 0) x = f.cell[c - 1][v] + (pick(2) ? 1 : -1) * (pick(2) ? 1e-10 : std::ldexp(1.0, -pick(60)));
      if (kind == 8 && pick(12) == 0) {
        const double bad[] = {0.0, -0.0, -x, INFINITY, -INFINITY, NAN, 1e300, 1e-310, -1e-310};
        x = bad[pick(9)];
      }
    }
  }
  return f;
}

int main()
{
  const int n = 1 << 16;
  std::vector<Face> h(n);
  Face* faces;
  int* count;
  if (cudaMalloc(&faces, n * sizeof(Face)) != cudaSuccess || cudaMalloc(&count, 3 * sizeof(int)) != cudaSuccess) return 2;
  int bad = 0;
  for (int kind = 0; kind < 9; ++kind) {
    for (Face& f : h) f = face(kind);
    if (cudaMemcpy(faces, h.data(), n * sizeof(Face), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    for (int s = 0; s < 3; ++s) {
      int c[3] = {0, 0, n};
      cudaMemcpy(count, c, sizeof c, cudaMemcpyHostToDevice);
      if (s == 0) compare<dn::AusmPlusFace><<<n / 128, 128>>>(faces, n, count, count + 1, count + 2);
      if (s == 1) compare<dn::VanLeerFace><<<n / 128, 128>>>(faces, n, count, count + 1, count + 2);
      if (s == 2) compare<dn::RoeFace><<<n / 128, 128>>>(faces, n, count, count + 1, count + 2);
      if (cudaMemcpy(c, count, sizeof c, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
      std::printf("%s %s %d %d", s == 0 ? "ausm" : s == 1 ? "vanleer" : "roe", kKinds[kind], c[0], c[1]);
      if (c[1]) {
        const Face& f = h[c[2]];
        std::printf("  first: dir %d sl %d sr %d A %a", f.dir, f.sl, f.sr, f.A);
        for (int q = 0; q < 4; ++q)
          for (int v = 0; v < 5; ++v) std::printf(" %a", f.cell[q][v]);
      }
      std::printf("\n");
      bad += c[1];
    }
  }
  return bad ? 1 : 0;
}
