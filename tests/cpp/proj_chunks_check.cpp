// The chunk tables of the projection kernels when a device allocation fails: the build
// reports it, a second call builds them again, and nothing is taken for built before all of
// it is there.  setup.cpp is compiled into this program with a fake CUDA allocator whose n-th
// allocation fails.
#include <cstdio>
#include <cstdlib>

#include "../../inq-wannier-fork_b200/csrc/setup.cpp"

static int g_fail_at = -1, g_calls = 0;
static cudaError_t g_last = cudaSuccess;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_calls++ == g_fail_at) return g_last = cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
namespace inqb {
size_t project_table_bytes(int, int chunks) { return (size_t)chunks * kProjChunk * 64; }
}

int main() {
  using namespace inqb;
  int bad = 0;
  for (int fail_at = 0; fail_at < 6; fail_at++) {
    ProjTables t;
    t.nproj = 2;
    t.L = 1;
    t.nent = 3;
    t.atom_ptr = {0, 2, 3};
    t.atom_ent = {0, 1, 2};
    t.ent_pt = {5, 6, 7};
    t.ent_beta = {1.0, 2.0, 3.0};
    t.ent_relpos.assign(9, 0.0f);
    inqb_ctx ctx;
    ctx.precision = INQB_FP64;
    g_calls = 0;
    g_fail_at = fail_at;
    const int st = build_proj_chunks(ctx, t);
    const bool fails = fail_at < 5;  // five device buffers
    bad += (st == INQB_OK) == fails;
    bad += fails && t.pc_chunks != 0;
    bad += cudaGetLastError() != cudaSuccess;  // the next launch check must not see it
    g_fail_at = -1;
    bad += build_proj_chunks(ctx, t) != INQB_OK;
    bad += t.pc_chunks != 2 || !t.d_pc_ptr.ptr || !t.d_pc_pt.ptr || !t.d_pc_beta.ptr || !t.d_pc_relpos.ptr;
    bad += !t.d_pc_table.ptr || t.d_pc_table.bytes < project_table_bytes(INQB_FP64, 2);
  }
  printf("bad=%d\n", bad);
  return bad != 0;
}
