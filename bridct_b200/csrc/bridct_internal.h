// Internal types shared by the host-side translation units of libbridct_b200.so.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "plain_launch.cuh"

namespace bridct {

// One per CUDA device, created on first use and immutable afterwards.
struct DeviceCtx {
  int device = 0;
  int sm_count = 0;
  int major = 0, minor = 0;
  LaunchCtx launch{};
  PlainLauncher plain[8][8][3] = {};
  SplitTables split[4] = {};            // rotation tables of N = 128, 256, 512, 1024
  std::vector<void*> table_mem;
  LineTables line_tables(int h, int w) const;
};

void set_error(const std::string& s);
int cuda_fail(cudaError_t e, const char* what);
double sj_scale(int n, int k);
// Copies a table to the device and waits until it has arrived.  A plain cudaMemcpy from pageable memory may
// return while the last part is still on its way, and the kernels that read the tables run on streams that
// do not wait for the default stream.
cudaError_t upload_table(void* dst, const void* src, size_t bytes);
// Rotation tables of the split lines of N = 128..1024 points (sj_split.cuh, SplitTab), float64-derived:
// their size, and their values to t.
int split_table_floats(int N);
void fill_split_tables(int N, float* t);
DeviceCtx* device_ctx(int device);

// One unit of a merged pass (merged.cu): a column strip or a row block, starting `off` floats into both
// x and y, rows ld floats apart, of lines of n points in the given mode.
struct MergedUnit {
  long long off;
  int ld;
  short n, mode;
};
// Which kernel takes the units of line length n (columns 0..2, rows 0..3), the strip width of column
// length h, the row-block height of row length w, and one such launch (columns x -> y, rows in place;
// mode -1: every unit in its own mode).
int merged_class(bool col, int n);
int merged_strip_cols(int h);
int merged_block_rows(int w);
cudaError_t launch_merged_pass(const DeviceCtx* d, bool col, int cls, int mode, const MergedUnit* units, long long n,
                               const float* x, float* y, cudaStream_t st);
// Opts `kernel` into `smem` bytes of dynamic shared memory on the current device and returns
// its resident blocks per SM at `threads` threads (0 on failure); cached per device, since the
// attribute belongs to the device's copy of the kernel.  all_shared: the kernel asks for the SM's largest
// shared-memory configuration.
int kernel_setup(const void* kernel, int smem, int threads, bool all_shared);
int current_device(int* dev);
const void* device_address(const void* p, bool* pinned);

// Makes `device` current for the guard's scope and gives the caller's current device back at
// scope exit, so an entry point never leaves another device current than the one it found.
struct DeviceGuard {
  int prev = -1;
  cudaError_t status = cudaSuccess;
  explicit DeviceGuard(int device) {
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess) {
      cudaGetLastError();
      cur = -1;
    }
    if (cur != device) {
      status = cudaSetDevice(device);
      prev = cur;
    }
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
  DeviceGuard(const DeviceGuard&) = delete;
  DeviceGuard& operator=(const DeviceGuard&) = delete;
};

}  // namespace bridct

struct bridct_plan {
  int h = 0, w = 0;
  size_t elements = 0;
  int square = 0;
  int device = 0;
  bridct::DeviceCtx* dev = nullptr;
  cudaStream_t stream = nullptr;
  float* d_x = nullptr;        // one-array device staging
  float* d_y = nullptr;
  float* pin = nullptr;        // one-array pinned staging (in, out)
  // batch pipeline (allocated on the first host-pointer batch call): copy-in, kernel and
  // copy-out streams, and per slot the events that order a slot's reuse on the GPU
  static constexpr int kPipeSlots = 4;
  cudaStream_t aux[3] = {nullptr, nullptr, nullptr};
  cudaEvent_t pipe_ev[3][kPipeSlots] = {};   // [copied in, transformed, copied out][slot]
  float* d_batch = nullptr;    // slots x (in, out) x chunk
  float* pin_batch = nullptr;  // slots x (in, out) x chunk, pageable callers only
  void* copyout = nullptr;     // per slot, the state of a pageable output's copy out (host_pipeline.cu)
  size_t chunk = 0;            // arrays per pipeline chunk
  // precision-form scratch (allocated on first use of a tensor-core form that is not given a
  // caller workspace); tc_mu serializes its (re)allocation
  void* tc_mem = nullptr;
  size_t tc_bytes = 0;
  std::mutex tc_mu;
};

namespace bridct {
// Pipeline-only mode: forward then inverse with the float32 spectrum materialized on the device
// (bitwise the composition of a FORWARD and an INVERSE call).
constexpr int kModeSpectrumRT = 3;
int launch_plain_form(const bridct_plan* p, int mode, const float* x, float* y, long long batch,
                      cudaStream_t st);
// Plain form over `batch` h x w arrays on device d in general layouts (lx, ly NULL: contiguous).
int launch_plain_layout(DeviceCtx* d, int h, int w, int mode, const float* x, float* y, long long batch,
                        const BatchLayout* lx, const BatchLayout* ly, cudaStream_t st);
int host_batch_pipeline(bridct_plan* p, int mode, const float* in, float* out, size_t batch,
                        const float* dx, float* dy, bool pin_in, bool pin_out);
bridct_plan* thread_square_plan(int n);
// memcpy split over the library's host copy threads (pageable <-> pinned staging).
void host_copy(void* dst, const void* src, size_t n);
void release_plan_extras(bridct_plan* p);
}  // namespace bridct

namespace bridct {
// Tensor-core precision forms (tc_forms.cu).
// workspace: caller-owned scratch of ws_bytes (NULL: the plan's own scratch).
int apply_tc_form(bridct_plan* p, int mode, int form, const float* x, float* y, size_t batch,
                  void* stream, void* workspace, size_t ws_bytes);
// Scratch bytes a tensor-core form needs for `batch` arrays of the plan's shape (0: none).
size_t tc_workspace_bytes(const bridct_plan* p, int form, size_t batch);
}  // namespace bridct
