// host_only.cu — the library's host code without its tile kernels, to be linked
// with host_runtime.cpp, a CUDA runtime that has no GPU behind it. What the host
// decides (tiles, copies, limits, allocations, error codes) can then be tested
// on any machine.
#include "../../opensayal_gb300/csrc/os_fluid.cu"
#include "host_only.h"

// ---------------------------------------------------------------------------
// The tile kernels: one function per instantiation, told apart by address.
// ---------------------------------------------------------------------------
namespace {

struct FakeKernel {
  const void* fn;
  int32_t kind;
};
std::vector<FakeKernel>& fake_kernels() {
  static std::vector<FakeKernel> v;
  return v;
}

template <int R, int FORM>
void fake_project(const osg::ProjectArgs) {
  static volatile int id;
  id = 64 * R + FORM;  // a body of its own, so that no two are folded
}
template <int R, int FORM>
void fake_diffuse(const osg::DiffuseArgs) {
  static volatile int id;
  id = 64 * R + FORM;
}
template <int PHASE>
void fake_batch(const osg::PlanHeader*, const int*, int, int, const osg::RegTile,
                const osg::ResidentSync) {
  static volatile int id;
  id = PHASE;
}

template <class Fn>
Fn known(Fn fn, int32_t kind) {
  for (const FakeKernel& k : fake_kernels())
    if (k.fn == reinterpret_cast<const void*>(fn)) return fn;
  fake_kernels().push_back({reinterpret_cast<const void*>(fn), kind});
  return fn;
}
template <int R>
osg::ProjectKernel fake_project_kernel(bool pressure, bool aligned) {
  osg::ProjectKernel fn = aligned ? (pressure ? fake_project<R, 3> : fake_project<R, 1>)
                                  : (pressure ? fake_project<R, 2> : fake_project<R, 0>);
  return known(fn, kProject);
}
template <int R>
osg::DiffuseKernel fake_diffuse_kernel(bool aligned) {
  osg::DiffuseKernel fn = aligned ? fake_diffuse<R, 1> : fake_diffuse<R, 0>;
  return known(fn, kDiffuse);
}

}  // namespace

namespace osg {
template <> ProjectKernel project_kernel<2>(bool p, bool a) { return fake_project_kernel<2>(p, a); }
template <> ProjectKernel project_kernel<4>(bool p, bool a) { return fake_project_kernel<4>(p, a); }
template <> ProjectKernel project_kernel<6>(bool p, bool a) { return fake_project_kernel<6>(p, a); }
template <> ProjectKernel project_kernel<8>(bool p, bool a) { return fake_project_kernel<8>(p, a); }
template <> ProjectKernel project_kernel<10>(bool p, bool a) { return fake_project_kernel<10>(p, a); }
template <> DiffuseKernel diffuse_kernel<2>(bool a) { return fake_diffuse_kernel<2>(a); }
template <> DiffuseKernel diffuse_kernel<4>(bool a) { return fake_diffuse_kernel<4>(a); }
template <> DiffuseKernel diffuse_kernel<6>(bool a) { return fake_diffuse_kernel<6>(a); }
template <> DiffuseKernel diffuse_kernel<8>(bool a) { return fake_diffuse_kernel<8>(a); }
template <> DiffuseKernel diffuse_kernel<12>(bool a) { return fake_diffuse_kernel<12>(a); }
BatchTileKernel batch_project_kernel() { return known(fake_batch<0>, kBatchProject); }
BatchTileKernel batch_diffuse_kernel() { return known(fake_batch<1>, kBatchDiffuse); }
}  // namespace osg

void describe_tile(const osg::RegTile& g, HostLaunch* l) {
  l->tiles = g.tiles_x * g.tiles_y, l->tiles_y = g.tiles_y;
  l->R = g.R, l->warps = g.warps, l->halo = g.halo;
}

// The arguments of a launch of these kernels.
extern "C" void host_describe(const void* fn, void** args, HostLaunch* l) {
  for (const FakeKernel& k : fake_kernels())
    if (k.fn == fn) l->kind = k.kind;
  if (l->kind == kProject) {
    const auto& a = *static_cast<const osg::ProjectArgs*>(args[0]);
    l->n = a.n, l->K = a.K, l->D = a.D;
    describe_tile(a.g, l);
    l->ui = a.ui, l->vi = a.vi, l->uo = a.uo, l->vo = a.vo;
    l->err = a.sync.dev_err;
  } else if (l->kind == kDiffuse) {
    const auto& a = *static_cast<const osg::DiffuseArgs*>(args[0]);
    l->n = a.n, l->K = a.K, l->D = a.D;
    describe_tile(a.g, l);
    l->ui = a.ui, l->uo = a.uo;
    l->err = a.sync.dev_err;
  }
}

extern "C" int32_t host_segment(int32_t projection, int32_t n, int32_t K, int32_t D,
                                int32_t storage, int32_t k, int32_t* messages, int32_t* round,
                                int32_t* exchange) {
  for (int done = 0; done < n; k--) {
    const osg::Segment s = osg::segment_at(n, K, D, done, storage);
    if (k == 0) {
      *messages = projection ? osg::project_messages(s.sweeps) : s.sweeps;
      *round = s.round, *exchange = s.exchange;
      return s.sweeps;
    }
    done += s.sweeps;
  }
  return 0;
}
