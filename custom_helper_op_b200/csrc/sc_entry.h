// Launch entry points of the manifold-convolution kernels.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace chop {
struct ScArgs;
int sc_fwd_simt_launch(int dtype, const ScArgs& a, cudaStream_t st);
int sc_dgrad_simt_launch(int dtype, const ScArgs& a, cudaStream_t st);
int sc_wgrad_simt_launch(int dtype, const ScArgs& a, cudaStream_t st);
int sc_tconv_simt_launch(int dtype, const ScArgs& a, cudaStream_t st);
int sc_twgrad_simt_launch(int dtype, const ScArgs& a, int nparts, cudaStream_t st);
int sc_pad_launch(int dtype, bool grad, const void* src, const int* base_plane, void* dst, int B, int h, int w, int d,
                  int C, int sr, int sc, int sd, cudaStream_t st);
int sc_wgrad_parts(long long nvox_out);
int sc_wgrad_simt_launch_parts(int dtype, const ScArgs& a, int nparts, cudaStream_t st);
int sc_static_scratch(void** ptr, size_t* bytes);
bool sc_umma_supported(int dtype, const ScArgs& a);
int sc_umma_fwd_launch(const ScArgs& a, cudaStream_t st);
int sc_umma_dgrad_launch(const ScArgs& a, cudaStream_t st);
int sc_umma_wgrad_launch(const ScArgs& a, int nparts, cudaStream_t st);
int sc_umma_twgrad_launch(const ScArgs& a, int nparts, cudaStream_t st);
bool sc_tile_supported(int dtype, const ScArgs& a);
int sc_tile_fwd_launch(int dtype, const ScArgs& a, cudaStream_t st);
int sc_tile_wgrad_launch(int dtype, const ScArgs& a, int nparts, cudaStream_t st);
int sc_tile_twgrad_launch(int dtype, const ScArgs& a, int nparts, cudaStream_t st);
int sc_tile_gather_launch(int dtype, const ScArgs& a, cudaStream_t st);
// float32, 3x3x3, stride 1, by runs of planes (sc_run.cu) or on the tensor cores (sc_band.cu); the filter may lie at any address
bool sc_run_supported(int dtype, const ScArgs& a, int gathered);
int sc_run_launch(const ScArgs& a, bool dgrad, cudaStream_t st);
bool sc_run_wgrad_supported(int dtype, const ScArgs& a);
int sc_run_wgrad_launch(const ScArgs& a, int nparts, cudaStream_t st);
// sums nparts slabs of taps*KC*NC + 1 floats; default_grad may be null
int sc_slab_reduce(const float* part, int nparts, int taps, int KC, int NC, bool transposed, float* filter_grad,
                   float* default_grad, cudaStream_t st);
// stride 1 with every voxel staged once per tile (sc_band.cu); cin: gathered channels, cout: produced ones
bool sc_band_better(const ScArgs& a, int cin, int cout);
int sc_band_launch(const ScArgs& a, bool dgrad, cudaStream_t st);
bool sc_band_f32_better(const ScArgs& a, int cin, int cout);
int sc_band_f32_launch(const ScArgs& a, bool dgrad, cudaStream_t st);   // float32, in three bfloat16 pieces
int sc_band_timeouts();
int sc_band_publish_mirror(int* dptr, cudaStream_t st);
int sc_band_clear_timeouts();
// strided gather form with every coarse voxel staged once (sc_up.cu)
bool sc_up_supported(int dtype, const ScArgs& a);
int sc_up_launch(const ScArgs& a, cudaStream_t st);
bool sc_up_f32_supported(int dtype, const ScArgs& a);   // float32, in three bfloat16 pieces; the filter may lie at any address
int sc_up_f32_launch(const ScArgs& a, cudaStream_t st);
int sc_up_timeouts();
int sc_up_publish_mirror(int* dptr, cudaStream_t st);
int sc_up_clear_timeouts();
int sc_umma_timeouts();
int sc_umma_watch();
int sc_umma_note_timeout_for_test(int on);
void sc_umma_set_rows(int on);
size_t sc_wgrad_workspace_bytes(int dtype, int taps, int Cin, int Cout, long long nvox_out);
}  // namespace chop
