// skg_internal.h -- declarations shared between the library's translation units.
#pragma once
#include "../../include/skirt_b200.h"
#include <cuda_runtime.h>
#include <cstdint>
#include <chrono>
#include <string>
#include <thread>
#include <vector>

namespace skg {

struct DevGrid;
struct DevScene;
struct RunParams;

// skg_trace.cu (compiled with --fmad=false: bit-exact FP64 traversal)
cudaError_t launch_count_segments(const DevGrid& g, const double* r, const double* k, int64_t n,
                                  int precision, int64_t* counts, unsigned* err, cudaStream_t s);
cudaError_t launch_write_segments(const DevGrid& g, const double* r, const double* k, int64_t n,
                                  int precision, const int64_t* offsets, int32_t* cells, double* ds,
                                  unsigned* err, cudaStream_t s);
cudaError_t launch_optical_depth(const DevGrid& g, const DevScene* dS, const double* r, const double* k,
                                 int64_t n, int ell, int precision, double* tau, unsigned* err,
                                 cudaStream_t s);

// skg_setup.cu
cudaError_t launch_sample_density(const DevGrid& g, const DevScene* dS, const void* dgeoms,
                                  const double* norms, int ncomp, int nsamples, uint64_t seed,
                                  double* rho, cudaStream_t s);
cudaError_t launch_node_mass(const void* dgeoms, const double* norms, int ncomp, const double* boxes,
                             int nnodes, int nsamples, uint64_t seed, uint64_t node_offset,
                             double* mass, double* rhomin, double* rhomax, cudaStream_t s);
cudaError_t launch_dust_emission(const DevGrid& g, const DevScene* dS, const double* Tv,
                                 const double* planckabs, int nT, double* tab /* [3 nlambda] */, double* emit_Lv,
                                 double* temperature, cudaStream_t s);
size_t emission_tiles(int ncells);
cudaError_t launch_emission_sources(int nlambda, int ncells, const double* emit_Lv, double* emit_cdf,
                                    double* emit_Ltot, double* sums /* [nlambda][emission_tiles] */, cudaStream_t s);
cudaError_t launch_cell_major(const double* in, int64_t nc, int nl, int64_t m0, int64_t n, double* out, cudaStream_t s);
cudaError_t launch_sum(const double* x, int64_t n, double* out, cudaStream_t s);
cudaError_t launch_octant_records(const DevGrid& g, void* out, cudaStream_t s);   // out: 16 uint4 per cell
// Voronoi lists per peel-off direction: padded counts per (group, cell) (cnt[ngroups * ncells] = 0), their
// exclusive sums, then the lists at those offsets
cudaError_t launch_group_counts(const DevGrid& g, const double* kx, const double* ky, const double* kz, int ngroups,
                                int* cnt, cudaStream_t s);
size_t offset_scan_scratch_bytes(int n);
cudaError_t launch_offset_scan(const int* cnt, int* first, int n, void* scratch, size_t scratch_bytes, cudaStream_t s);
cudaError_t launch_group_planes(const DevGrid& g, const double* kx, const double* ky, const double* kz, int ngroups,
                                const int* first, void* planes, void* nexts, void* ranges, cudaStream_t s);
cudaError_t launch_embed_density(const DevGrid& g, const float* rhof, cudaStream_t s);

// skg_host.cpp
void sersic_table(double n, double* sv, double* Sv, double* Mv);      // 101 points each
void chunk_params(double packages, int nthreads, int nprocs, int nlambda,
                  uint64_t& nchunks, uint64_t& chunksize, uint64_t& npp);

// Between two looks at the device: nothing for the first 2 ms of a wait (a sleep of 50 us lasts about 100,
// and the smallest phases take less than 1 ms: 10^4 packets 1.20 against 1.25 ms a pass), then `us` of sleep.
inline void wait_a_little(std::chrono::steady_clock::time_point since, int us) {
    if (std::chrono::steady_clock::now() - since < std::chrono::milliseconds(2)) std::this_thread::yield();
    else std::this_thread::sleep_for(std::chrono::microseconds(us));
}

// error message of the calling thread
void set_error(const std::string& msg);
const char* get_error();

}  // namespace skg
