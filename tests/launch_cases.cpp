// Cases of test_launch_cpu.py: the library's launch code on fake_cudart.h.
#include "fake_cudart.h"
#include "ffg_internal.h"

using namespace ffg;

namespace ffg {
int launch_nedelec_oriented(const Topology &, const OrientedTables &, const DeviceTopology &,
                            const AssemblyInputs &, double *, double *, int *, cudaStream_t, bool) {
  return FFG_OK;
}
DeviceArena::~DeviceArena() {}
void *DeviceArena::take(size_t bytes) { return std::malloc(bytes); }
}  // namespace ffg

namespace {

// `rows` rows of `width` entries, 148 CTAs.
struct System {
  DeviceSell A;
  SolveWork w;
  std::vector<double> x, b;
  System(int64_t rows, int width) : x(rows), b(rows) {
    A.n = rows;
    A.n_slices = (rows + kSliceRows - 1) / kSliceRows;
    A.grid = 148;
    std::vector<int64_t> soff(A.n_slices + 1);
    for (int64_t s = 0; s <= A.n_slices; ++s) soff[s] = s * kSliceRows * width;
    A.padded = soff.back();
    std::vector<int> cs, ws, wo;
    sell_partition(soff.data(), A.n_slices, A.grid, cs, ws, wo);
    CHECK(sell_shares(soff.data(), cs, A) == FFG_OK);
    static int16_t dcol[1];
    A.dcol = dcol;
    CHECK(solve_work_alloc(w, rows, A.grid) == FFG_OK);
  }
};

struct Batch {
  std::vector<const DeviceSell *> A;
  std::vector<const double *> b;
  std::vector<double *> x;
  std::vector<SolveWork *> w;
  explicit Batch(std::vector<System> &s) {
    for (auto &k : s) {
      A.push_back(&k.A);
      b.push_back(k.b.data());
      x.push_back(k.x.data());
      w.push_back(&k.w);
    }
  }
};

ffg_solver_options options(int precision) {
  ffg_solver_options o;
  std::memset(&o, 0, sizeof(o));
  o.precision = precision;
  o.tolerance = 1e-10;
  o.max_iterations = 100;
  return o;
}

bool named(const Launch &l, const char *part) { return l.name.find(part) != std::string::npos; }

// A wait that ran out is seen by whichever CTA it ran out in: that CTA writes
// the control word, the first CTA may still have reported convergence.
void batch_reports_a_wait_that_ran_out(int precision) {
  std::vector<System> s;
  for (int k = 0; k < 3; ++k) s.emplace_back(1000 + 500 * k, 7);
  Batch B(s);
  on_launch = [&](const Launch &l, void **) {
    if (!named(l, "pcg_")) return;
    for (auto &k : s) {
      k.w.control[0] = 0;  // the kernels' first store
      k.w.result[0] = 1.0;
    }
    s[1].w.control[0] = FFG_TIMEOUT;
  };
  std::string msg;
  for (int rep = 0; rep < 2; ++rep) {
    CHECK(pcg_launch_batch(3, B.A.data(), B.b.data(), B.x.data(), options(precision), B.w.data(), 0,
                           msg) == FFG_OK);
    ffg_solver_stats st;
    CHECK(pcg_collect(s[0].w, &st, msg) == FFG_OK && st.converged);
    CHECK(pcg_collect(s[1].w, &st, msg) == FFG_TIMEOUT);
    CHECK(pcg_collect(s[2].w, &st, msg) == FFG_OK && st.converged);
  }
}

// Systems that fit the grid together share one launch, in every precision.
void groups_side_by_side(int precision, int64_t rows, int width) {
  std::vector<System> s;
  for (int k = 0; k < 3; ++k) s.emplace_back(rows + 500 * k, width);
  Batch B(s);
  std::string msg;
  CHECK(pcg_launch_groups(3, B.A.data(), B.b.data(), B.x.data(), options(precision), B.w.data(), 0,
                          msg) == FFG_OK);
  CHECK(launches.size() == 1 && launches[0].cooperative && launches[0].blocks <= 148);
}

struct Mesh {
  Topology t;
  ElementTables tab;
  DeviceTopology dt;
  DeviceSell A;
  AssemblyInputs in;
  int2 range[1];
  Mesh(int family, int nb, int max_column) {
    t.family = family;
    t.nb = nb;
    t.device_free = 100;
    t.max_column = max_column;
    A.n = 100;
    A.n_slices = 4;
    A.inc_range = range;
  }
  int columns() {
    return launch_columns(t, tab, dt, in, nullptr, 8, nullptr, nullptr, nullptr, nullptr, &A,
                          nullptr, nullptr, 0);
  }
  int batch() {
    AsmSys s;
    s.nb = t.nb;
    s.n_free = 100;
    s.max_width = t.max_column;
    return launch_batch_assembly(t.family, 1, &s, 0);
  }
};

// Another thread assembles a mesh of shorter columns between this one's calls
// to the runtime.
void assembly_beside_another(int family, int nb, bool batch) {
  Mesh big(family, nb, 200), small(family, nb, 9);
  auto go = [&](Mesh &m) { return batch ? m.batch() : m.columns(); };
  bool inside = false;
  on_attribute = [&](const void *) {
    if (inside) return;
    inside = true;
    CHECK(go(small) == FFG_OK);
    inside = false;
  };
  CHECK(go(big) == FFG_OK);
  int slices = 0;
  for (const Launch &l : launches) slices += named(l, "slice_kernel");
  CHECK(slices == 2);
}

// The cell kernel of an adjoint of this order: true when its launch was accepted.
bool adjoint(int order) {
  Topology t;
  ElementTables tab;
  DeviceTopology dt;
  DeviceArena scratch;
  t.family = FFG_TETRA_NEDELEC;
  t.degree = order;
  t.nb = order * (order + 2) * (order + 3) / 2;
  t.n_cells = 1;
  tab.n_terms = 12;
  double elem[1];
  struct Launched {};
  on_launch = [](const Launch &l, void **) {
    if (named(l, "nedelec_cell_vjp")) throw Launched();
  };
  try {
    nedelec_vjp(t, tab, dt, nullptr, nullptr, nullptr, nullptr, 1, 1, elem, nullptr, nullptr,
                nullptr, 0, scratch);
  } catch (Launched) {
    return true;
  }
  return false;
}

void adjoints_of_different_orders() {
  bool inside = false;
  on_attribute = [&](const void *) {
    if (inside) return;
    inside = true;
    CHECK(adjoint(6));
    inside = false;
  };
  CHECK(adjoint(5));
}

}  // namespace

int main(int argc, char **argv) {
  const std::string which = argc > 1 ? argv[1] : "";
  if (which == "batch_status_cluster") batch_reports_a_wait_that_ran_out(FFG_PRECISION_MIXED);
  else if (which == "batch_status_single") batch_reports_a_wait_that_ran_out(FFG_PRECISION_MIXED16);
  else if (which == "threads_p1") assembly_beside_another(FFG_TRIANGLE_P1, 3, false);
  else if (which == "threads_p2") assembly_beside_another(FFG_TETRA_LAGRANGE, 10, false);
  else if (which == "threads_nedelec") assembly_beside_another(FFG_TETRA_NEDELEC, 45, false);
  else if (which == "threads_batch") assembly_beside_another(FFG_TETRA_LAGRANGE, 10, true);
  else if (which == "threads_adjoint") adjoints_of_different_orders();
  else if (which == "groups_fp64") groups_side_by_side(FFG_PRECISION_FP64, 17000, 7);
  else if (which == "groups_mixed") groups_side_by_side(FFG_PRECISION_MIXED, 17000, 7);
  else if (which == "groups_large") groups_side_by_side(FFG_PRECISION_MIXED, 490000, 28);
  else if (which == "groups_mixed16") groups_side_by_side(FFG_PRECISION_MIXED16, 17000, 7);
  else return 2;
  return 0;
}
