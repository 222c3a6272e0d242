// The device's vector operations for the 3D Newton driver (newton3d.cuh): vectors of
// the canvas length N = nvar * cells in one workspace, basis vector i at V(i).
#pragma once
#include <vector>

#include "device3d.cuh"
#include "newton3d.cuh"

namespace jr {

// The scalars a GMRES cycle keeps on the device: the dots of the two orthogonalisations, the
// Hessenberg matrix (row-major, m + 1 rows of m), 1 / |w|, the reductions' ticket (0 between
// kernels) and the physicality flag.
struct Gmres3 {
  double h1[MAX_RESTART3 + 1], h2[MAX_RESTART3 + 1], H[(MAX_RESTART3 + 1) * MAX_RESTART3], inv;
  unsigned ticket;
  int flag;
};

struct DeviceOps3 {
  enum { R_ = 0, Z_, W_, T_, RES_, B_, DU_, ACT_, BASE };
  Plan3Dev p;
  size_t N = 0, n = 0;
  void* A = nullptr;                 // the primitive canvas of the residual / J.v (Dual-sized)
  void* factor = nullptr;            // the line factor (computed in prepare when line)
  bool line = false;
  // the linearised J.v's buffers (linearize3d.cuh); null where they did not fit the device's
  // memory: the products are then evaluated by the dual-number J.v
  double *lin_face = nullptr, *lin_cell = nullptr, *lin_dq = nullptr;
  double* vecs = nullptr;
  double* vdt = nullptr;
  double* partial = nullptr;
  Gmres3* gm = nullptr;
  int* flag = nullptr;
  double last_second = 0.0;
  cudaStream_t st = nullptr;

  int V(int i) const { return BASE + i; }
  double* v(int id) const { return vecs + (size_t)id * N; }
  double host_sum(int count, int halves);
  void prepare(const double* U, double cfl);
  void residual(const double* U, int out);
  void matvec(const double* U, double cfl, int src, int out);
  void precondition(const double* U, double cfl, int src, int dst);
  double dot(int a, int b);
  double nrm2(int a) { return sqrt(dot(a, a)); }
  void axpy(double al, int x, int y);
  void scale(double al, int x, int y);
  void copy(int x, int y);
  void zero(int y);
  double density_norm(int r);
  double worst_ratio(const double* U, int du);
  bool physical_after(const double* U, int du);
  void add_to_state(double* U, int du);
  static size_t work_doubles(size_t N, size_t n, int m);
  void bind(double* work, Gmres3* scalars, int m);
};

// the gmres3 newton_step3 (newton3d.cuh) finds for DeviceOps3
int gmres3(DeviceOps3& ops, const double* U, double cfl, const Newton3Config& c, int B, int X, int ACTION);

double newton_step3_device(DeviceOps3& ops, double* U, double& cfl, double& res_prev, const Newton3Config& c);

}  // namespace jr
