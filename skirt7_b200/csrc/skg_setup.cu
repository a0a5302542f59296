// skg_setup.cu -- set-up kernels: cell density sampling, tree-node mass sampling, the dust
// emission spectra (equilibrium temperature + grey body) and the per-wavelength cell CDFs from
// which dust packets are launched.
#include "skg_scene.cuh"
#include "skg_internal.h"
#include <cub/device/device_scan.cuh>

namespace skg {

// DustSystem::setSampleDensityBody (DustSystem.cpp:145-172): the density of a cell is the average
// of Nrandom samples of sum_h norm_h rho_h(r) at random positions in the cell.  One thread per cell.
__global__ void sample_density_kernel(const DevGrid g, const DevGeometry* __restrict__ geoms,
                                      const double* __restrict__ norms, int ncomp, int ns, uint64_t seed,
                                      double* rho) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= g.ncells) return;
    Philox rng;
    rng.init(seed, (uint64_t)m, 0x00D5u);
    double sum[MAX_COMP] = {0, 0, 0, 0};
    for (int n = 0; n < ns; n++) {
        V3<double> p = random_position_in_cell(g, m, rng);
        for (int h = 0; h < ncomp; h++) sum[h] += norms[h] * geom_density(geoms[h], p.x, p.y, p.z);
    }
    for (int h = 0; h < ncomp; h++) rho[(size_t)h * g.ncells + m] = sum[h] / ns;
}

cudaError_t launch_sample_density(const DevGrid& g, const DevScene*, const void* dgeoms, const double* norms,
                                  int ncomp, int nsamples, uint64_t seed, double* rho, cudaStream_t s) {
    int th = 128;
    int bl = (g.ncells + th - 1) / th;
    if (bl == 0) return cudaSuccess;
    sample_density_kernel<<<bl, th, 0, s>>>(g, (const DevGeometry*)dgeoms, norms, ncomp, nsamples, seed, rho);
    return cudaGetLastError();
}

// TreeNodeSampleDensityCalculator (TreeNodeSampleDensityCalculator.cpp:26-80): Nrandom random
// positions in a node box; mass = mean density x volume, plus the min/max sample for the density
// dispersion criterion.  One warp per node, lanes split the samples.
__global__ void node_mass_kernel(const DevGeometry* __restrict__ geoms, const double* __restrict__ norms, int ncomp,
                                 const double* __restrict__ boxes, int nnodes, int ns, uint64_t seed,
                                 uint64_t node_offset, double* mass, double* rmin, double* rmax) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (warp >= nnodes) return;
    const double* b = boxes + 6 * (size_t)warp;
    double sum = 0, lo = DBL_MAX, hi = 0;
    for (int n = lane; n < ns; n += 32) {
        Philox rng;
        rng.init(seed, node_offset + warp, 0x7EE0000u + n);
        double x = rng.uniform(), y = rng.uniform(), z = rng.uniform();
        x = b[0] + x * (b[3] - b[0]); y = b[1] + y * (b[4] - b[1]); z = b[2] + z * (b[5] - b[2]);
        double rho = 0;
        for (int h = 0; h < ncomp; h++) rho += norms[h] * geom_density(geoms[h], x, y, z);
        sum += rho; lo = fmin(lo, rho); hi = fmax(hi, rho);
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        lo = fmin(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
        double vol = (b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2]);
        mass[warp] = sum / ns * vol;
        rmin[warp] = lo; rmax[warp] = hi;
    }
}

cudaError_t launch_node_mass(const void* dgeoms, const double* norms, int ncomp, const double* boxes,
                             int nnodes, int nsamples, uint64_t seed, uint64_t node_offset,
                             double* mass, double* rhomin, double* rhomax, cudaStream_t s) {
    if (nnodes <= 0) return cudaSuccess;
    int th = 256;
    int bl = (int)(((int64_t)nnodes * 32 + th - 1) / th);
    node_mass_kernel<<<bl, th, 0, s>>>((const DevGeometry*)dgeoms, norms, ncomp, boxes, nnodes, nsamples, seed,
                                       node_offset, mass, rhomin, rhomax);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Dust emission spectra (one dust component, grey-body emissivity, every cell its own library
// entry: AllCellsDustLib + GreyBodyDustEmissivity).  Per cell:
//   J_ell = Labs(m,ell) / (kappa_abs rho 4 pi V) / dlambda            DustSystem.cpp:911-931
//   T     = invplanckabs( sum_ell kappa_abs J dlambda )                DustMix.cpp:674-697
//   L_ell = kappa_abs(ell) B_ell(T) dlambda, normalised to unit sum     GreyBodyDustEmissivity.cpp:21-45,
//                                                                       DustLib.cpp:135-148
// The mix's 1/mu factors cancel between the Planck table and the sum, as in the reference.

// Per wavelength, from the mix: tab[ell] = kappa_abs 2 h c^2 / lambda^5 dlambda and tab[nl + ell] =
// h c / (lambda k), so that L_ell = tab[ell] / (exp(tab[nl + ell] / T) - 1) (PlanckFunction.cpp:24-33); and
// tab[2 nl + ell] = 1 where the wavelength counts for the absorbed energy, 0 where J is not finite.
__global__ void planck_table_kernel(const DevScene* __restrict__ Sp, double* tab) {
    const DevScene& S = *Sp;
    const double h = 6.62606957e-34, c = 2.99792458e8, k = 1.3806488e-23;
    for (int ell = blockIdx.x * blockDim.x + threadIdx.x; ell < S.nlambda; ell += gridDim.x * blockDim.x) {
        const double lambda = S.lambda[ell], kabs = S.kext[ell] * (1.0 - S.albedo[ell]);
        tab[ell] = kabs * (2.0 * h * c * c / pow(lambda, 5)) * S.dlambda[ell];
        tab[S.nlambda + ell] = h * c / (lambda * k);
        tab[2 * S.nlambda + ell] = (kabs > 0.0 && S.dlambda[ell] != 0.0) ? 1.0 : 0.0;
    }
}

SKG_D double cell_volume(const DevGrid& g, int m) {
    if (g.type == SKG_GRID_CARTESIAN) {
        int i = m / (g.nz * g.ny), j = (m / g.nz) % g.ny, k = m % g.nz;
        return (g.xv[i + 1] - g.xv[i]) * (g.yv[j + 1] - g.yv[j]) * (g.zv[k + 1] - g.zv[k]);
    } else if (g.type == SKG_GRID_VORONOI) {
        return g.vvol[m];
    }
    const double* b = g.node_box + 6 * (size_t)g.cell_node[m];
    return (b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2]);
}

// Temperature of every cell and its luminosity per wavelength, emit_Lv[ell][m] = Labsbol[m] L_ell
// (PanMonteCarloSimulation.cpp:197-203).  One thread per cell; the spectrum is formed twice, once for
// its sum and once for the result: with the wavelengths' constants in a table an entry costs an exp and a division, less than
// writing the spectra out and reading them back twice (a pow and three divisions per entry
// before: 4.2 ms per call for 10^6 cells and 40 wavelengths, with the sums below).
__global__ void __launch_bounds__(128) dust_emission_kernel(const DevGrid g, const DevScene* __restrict__ Sp,
                                                            const double* __restrict__ Tv,
                                                            const double* __restrict__ planckabs, int nT,
                                                            const double* __restrict__ tab, double* __restrict__ emit_Lv,
                                                            double* temperature) {
    const DevScene& S = *Sp;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= S.ncells) return;
    const int nl = S.nlambda;
    const size_t nc = (size_t)S.ncells;
    const double* const ls = S.labs_stel + m;
    const double* const ld = S.labs_dust + m;
    double lb = 0, la = 0;
#pragma unroll 4
    for (int ell = 0; ell < nl; ell++) {
        const double v = ls[ell * nc] + ld[ell * nc];
        lb += v;
        la += v * __ldg(tab + 2 * nl + ell);
    }
    const double q = S.rho[m] * (4.0 * M_PI * cell_volume(g, m));
    double pa = la / q;                            // sum of kappa_abs J dlambda
    if (!isfinite(pa)) pa = 0.0;
    const int p = dlocate_clip(planckabs, nT, pa);
    const double T = Tv[p] + ((pa - planckabs[p]) / (planckabs[p + 1] - planckabs[p])) * (Tv[p + 1] - Tv[p]);
    if (temperature) temperature[m] = T;
    double total = 0;
    const double invT = 1.0 / T;
    if (T > 0)
        for (int ell = 0; ell < nl; ell++) total += __ldg(tab + ell) / (exp(__ldg(tab + nl + ell) * invT) - 1.0);
    const double f = (total > 0 && lb > 0.0) ? lb / total : 0.0;
    for (int ell = 0; ell < nl; ell++)
        emit_Lv[ell * nc + m] = f > 0 ? f * (__ldg(tab + ell) / (exp(__ldg(tab + nl + ell) * invT) - 1.0)) : 0.0;
}

cudaError_t launch_dust_emission(const DevGrid& g, const DevScene* dS, const double* Tv, const double* planckabs,
                                 int nT, double* tab, double* emit_Lv, double* temperature, cudaStream_t s) {
    int th = 128;
    int bl = (g.ncells + th - 1) / th;
    if (bl == 0) return cudaSuccess;
    planck_table_kernel<<<1, 128, 0, s>>>(dS, tab);
    dust_emission_kernel<<<bl, th, 0, s>>>(g, dS, Tv, planckabs, nT, tab, emit_Lv, temperature);
    return cudaGetLastError();
}

// The cumulative cell luminosities, normalised per wavelength (NR::cdf, NR.hpp:388-394: P_0 = 0,
// P_{i+1} = sum_{j<=i} p_j / sum p): sums of tiles of cells, their offsets per wavelength, then the
// tiles again with their offset and the normalisation -- three launches for all wavelengths, the
// luminosities read twice and the result written once (a library scan per wavelength and a pass to
// normalise before: 80 launches for 40 wavelengths).  The last entry is 1.  The others are sums in more than one
// order (lanes, warps, tiles), so where cells without luminosity follow, an entry may lie a rounding below the one
// before it; deviates are multiples of 2^-33, some 10^6 times as far apart.
constexpr int CDF_TILE = 2048;                     // 8 warps of 8 rows of 32 cells
SKG_D double warp_incl(double v, int lane) {
    for (int d = 1; d < 32; d <<= 1) { const double t = __shfl_up_sync(0xffffffffu, v, d); if (lane >= d) v += t; }
    return v;
}
__global__ void __launch_bounds__(256) cdf_sums_kernel(int nc, const double* __restrict__ Lv, double* sums) {
    __shared__ double ws[8];
    const double* x = Lv + (size_t)blockIdx.y * nc;
    double v = 0;
    for (int i = 0; i < CDF_TILE / 256; i++) {
        const int64_t m = (int64_t)blockIdx.x * CDF_TILE + i * 256 + threadIdx.x;
        if (m < nc) v += x[m];
    }
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) v += ws[w];
        sums[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = v;
    }
}
// one block per wavelength: the tiles' sums become their offsets
__global__ void __launch_bounds__(256) cdf_offsets_kernel(int ntiles, double* sums, double* Ltot) {
    __shared__ double ws[8], carry;
    double* x = sums + (size_t)blockIdx.x * ntiles;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    for (int b = 0; b < ntiles; b += 256) {
        const int i = b + threadIdx.x;
        const double v = i < ntiles ? x[i] : 0.0;
        const double inc = warp_incl(v, lane);
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        double before = carry;
        for (int w = 0; w < warp; w++) before += ws[w];
        if (i < ntiles) x[i] = before + (inc - v);
        __syncthreads();
        if (threadIdx.x == 255) carry = before + inc;
        __syncthreads();
    }
    if (threadIdx.x == 0) Ltot[blockIdx.x] = carry;
}
__global__ void __launch_bounds__(256) cdf_kernel(int nc, const double* __restrict__ Lv, const double* __restrict__ offsets,
                                                  const double* __restrict__ Ltot, double* __restrict__ cdf) {
    __shared__ double ws[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ell = blockIdx.y;
    const double* x = Lv + (size_t)ell * nc;
    double* out = cdf + (size_t)ell * (nc + 1);
    const int64_t m0 = (int64_t)blockIdx.x * CDF_TILE + warp * (CDF_TILE / 8) + lane;
    double v[8];
    double sum = 0;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int64_t m = m0 + 32 * r;
        v[r] = sum + warp_incl(m < nc ? x[m] : 0.0, lane);
        sum = __shfl_sync(0xffffffffu, v[r], 31);
    }
    if (lane == 0) ws[warp] = sum;
    __syncthreads();
    double before = offsets[(size_t)ell * gridDim.x + blockIdx.x];
    for (int w = 0; w < warp; w++) before += ws[w];
    const double tot = Ltot[ell];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int64_t m = m0 + 32 * r;
        if (m < nc) out[m + 1] = !(tot > 0) ? 0.0 : m == nc - 1 ? 1.0 : fmin((before + v[r]) / tot, 1.0);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = 0.0;
}

size_t emission_tiles(int nc) { return ((size_t)nc + CDF_TILE - 1) / CDF_TILE; }

cudaError_t launch_emission_sources(int nl, int nc, const double* emit_Lv, double* emit_cdf, double* emit_Ltot,
                                    double* sums, cudaStream_t s) {
    if (nc <= 0 || nl <= 0) return cudaSuccess;
    const int tiles = (int)emission_tiles(nc);
    for (int l0 = 0; l0 < nl; l0 += 65535) {
        const int n = std::min(nl - l0, 65535);
        const double* x = emit_Lv + (size_t)l0 * nc;
        double* t = sums + (size_t)l0 * tiles;
        cdf_sums_kernel<<<dim3(tiles, n), 256, 0, s>>>(nc, x, t);
        cdf_offsets_kernel<<<n, 256, 0, s>>>(tiles, t, emit_Ltot + l0);
        cdf_kernel<<<dim3(tiles, n), 256, 0, s>>>(nc, x, t, emit_Ltot + l0, emit_cdf + (size_t)l0 * (nc + 1));
    }
    return cudaGetLastError();
}

// Writes each leaf's (single-component) density into its rope-tree record, so that a cell step
// of the FP32 walk reads box, density and ropes in one 64-byte gather.
__global__ void embed_density_kernel(float4* lrec, int nleaves, const float* __restrict__ rhof) {
    int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= nleaves) return;
    int cell = __float_as_int(lrec[4 * (size_t)li + 1].w);
    lrec[4 * (size_t)li].w = rhof[cell];
}
// The same for the lattice form: word 0 of cell m's 32-byte record.
__global__ void embed_density_lattice_kernel(uint4* prec, int ncells, const float* __restrict__ rhof) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= ncells) return;
    prec[2 * (size_t)m].x = __float_as_uint(rhof[m]);
}
// And the density of the neighbour behind each Voronoi wall: all of cell m's entries, padding included.
__global__ void embed_density_voronoi_kernel(const int2* __restrict__ ranges, int4* next, int ncells,
                                             const float* __restrict__ rhof) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= ncells) return;
    const int2 o = ranges[m];
    for (int q = o.x; q < o.y; q++) {
        const int mi = next[q].x;
        if (mi >= 0) next[q].w = __float_as_int(rhof[mi]);
    }
}
cudaError_t launch_embed_density(const DevGrid& g, const float* rhof, cudaStream_t s) {
    int n = g.ncells;
    if (n <= 0) return cudaSuccess;
    if (g.vnext) {
        embed_density_voronoi_kernel<<<(n + 127) / 128, 128, 0, s>>>(g.vpoff, const_cast<int4*>(g.vnext), n, rhof);
        return cudaGetLastError();
    }
    if (g.lattice) embed_density_lattice_kernel<<<(n + 255) / 256, 256, 0, s>>>(const_cast<uint4*>(g.prec), n, rhof);
    else embed_density_kernel<<<(n + 255) / 256, 256, 0, s>>>(const_cast<float4*>(g.lrec), n, rhof);
    return cudaGetLastError();
}

// The octant records of a lattice tree from its leaf records (density embedded): for octant o of the
// direction (bit a set: k_a < 0) and cell m, record o * ncells + m holds the walls ahead on x, y, z,
// the density, and the ropes of those walls (a record of the same octant, -1 outside, <= -2 an
// internal record).
__global__ void octant_records_kernel(const DevGrid g, uint4* out) {
    using L = TreeLatticeStepper<float>;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= g.ncells) return;
    L st;
    st.load(g, m);
    const uint32_t c[3] = {L::code_x(st.a), L::code_y(st.a), L::code_z(st.a)};
    for (int o = 0; o < 8; o++) {
        uint32_t w[3], r[3];
        for (int a = 0; a < 3; a++) {
            const bool up = !(o >> a & 1);
            w[a] = __float_as_uint(L::wall(c[a], up, g.lorg[a], g.lunit[a]));
            const int rp = st.rope(2 * a + (up ? 1 : 0));
            r[a] = (uint32_t)(rp >= 0 ? rp + o * g.ncells : rp);
        }
        uint4* p = out + 2 * ((size_t)o * g.ncells + m);
        p[0] = make_uint4(w[0], w[1], w[2], st.a.x);
        p[1] = make_uint4(r[0], r[1], r[2], 0);
    }
}
cudaError_t launch_octant_records(const DevGrid& g, void* out, cudaStream_t s) {
    octant_records_kernel<<<(g.ncells + 127) / 128, 128, 0, s>>>(g, (uint4*)out);
    return cudaGetLastError();
}

// The planes ahead of a peel-off direction, per cell: n.k > 0, formed as the walk forms it.
struct GroupDirs { float kx[4], ky[4], kz[4]; };
static GroupDirs group_dirs(const double* kx, const double* ky, const double* kz, int n) {
    GroupDirs d = {};
    for (int q = 0; q < n && q < 4; q++) { d.kx[q] = (float)kx[q]; d.ky[q] = (float)ky[q]; d.kz[q] = (float)kz[q]; }
    return d;
}
__global__ void group_counts_kernel(const DevGrid g, const GroupDirs d, int ngroups, int* cnt) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t > (int64_t)ngroups * g.nsites) return;
    int c = 0;
    if (t < (int64_t)ngroups * g.nsites) {
        const int q = (int)(t / g.nsites), m = (int)(t - (int64_t)q * g.nsites);
        const int2 o = g.vpoff[m];
        for (int i = o.x; i < o.y; i++) {
            const float4 p = g.vplane[i];
            c += vor_den(p.x, p.y, p.z, d.kx[q], d.ky[q], d.kz[q]) > 0.f;
        }
    }
    cnt[t] = (c + 1) & ~1;
}
__global__ void group_planes_kernel(const DevGrid g, const GroupDirs d, int ngroups, const int* __restrict__ first,
                                    float4* planes, int4* nexts, int2* ranges) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)ngroups * g.nsites) return;
    const int q = (int)(t / g.nsites), m = (int)(t - (int64_t)q * g.nsites);
    const int2 o = g.vpoff[m];
    const int end = first[t + 1];
    int at = first[t];
    ranges[t] = make_int2(at, end);
    for (int i = o.x; i < o.y; i++) {
        const float4 p = g.vplane[i];
        if (!(vor_den(p.x, p.y, p.z, d.kx[q], d.ky[q], d.kz[q]) > 0.f)) continue;
        const int4 nx = g.vnext[i];
        planes[at] = p;
        const int64_t f = (int64_t)q * g.nsites + max(nx.x, 0);
        const int np = first[f + 1] - first[f];
        nexts[at] = nx.x < 0 ? nx : make_int4(nx.x, first[f], nx.z == -1 ? -1 : np | (nx.z & ~0xffff), nx.w);
        at++;
    }
    for (; at < end; at++) { planes[at] = make_float4(0.f, 0.f, 0.f, 0.f); nexts[at] = make_int4(-1, 0, 0, 0); }
}
cudaError_t launch_group_counts(const DevGrid& g, const double* kx, const double* ky, const double* kz, int ngroups,
                                int* cnt, cudaStream_t s) {
    const int64_t n = (int64_t)ngroups * g.nsites + 1;
    group_counts_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(g, group_dirs(kx, ky, kz, ngroups), ngroups, cnt);
    return cudaGetLastError();
}
size_t offset_scan_scratch_bytes(int n) {
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const int*)nullptr, (int*)nullptr, n);
    return bytes;
}
cudaError_t launch_offset_scan(const int* cnt, int* first, int n, void* scratch, size_t scratch_bytes, cudaStream_t s) {
    return cub::DeviceScan::ExclusiveSum(scratch, scratch_bytes, cnt, first, n, s);
}
cudaError_t launch_group_planes(const DevGrid& g, const double* kx, const double* ky, const double* kz, int ngroups,
                                const int* first, void* planes, void* nexts, void* ranges, cudaStream_t s) {
    const int64_t n = (int64_t)ngroups * g.nsites;
    group_planes_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(g, group_dirs(kx, ky, kz, ngroups), ngroups, first,
                                                                    (float4*)planes, (int4*)nexts, (int2*)ranges);
    return cudaGetLastError();
}

// out[m - m0][ell] = in[ell][m] for the cells m0 .. m0 + n - 1: tiles of 32 cells x 32 wavelengths through
// shared memory, both sides coalesced.
__global__ void __launch_bounds__(256) cell_major_kernel(const double* __restrict__ in, int64_t nc, int nl, int64_t m0,
                                                         int64_t n, double* __restrict__ out) {
    __shared__ double t[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * 32;
    for (int e0 = 0; e0 < nl; e0 += 32) {
        for (int r = y; r < 32; r += 8)
            if (e0 + r < nl && c0 + x < n) t[r][x] = in[(size_t)(e0 + r) * nc + m0 + c0 + x];
        __syncthreads();
        for (int r = y; r < 32; r += 8)
            if (e0 + x < nl && c0 + r < n) out[(size_t)(c0 + r) * nl + e0 + x] = t[x][r];
        __syncthreads();
    }
}
cudaError_t launch_cell_major(const double* in, int64_t nc, int nl, int64_t m0, int64_t n, double* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    cell_major_kernel<<<(unsigned)((n + 31) / 32), 256, 0, s>>>(in, nc, nl, m0, n, out);
    return cudaGetLastError();
}

// Sum of a vector (absorbed-luminosity totals for the self-absorption convergence test).
__global__ void sum_kernel(const double* __restrict__ x, int64_t n, double* out) {
    __shared__ double sh[256];
    double acc = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) acc += x[i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) { if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o]; __syncthreads(); }
    if (threadIdx.x == 0) atomicAdd(out, sh[0]);
}
cudaError_t launch_sum(const double* x, int64_t n, double* out, cudaStream_t s) {
    cudaMemsetAsync(out, 0, sizeof(double), s);
    int bl = (int)std::min<int64_t>(1184, (n + 255) / 256);
    if (bl <= 0) return cudaSuccess;
    sum_kernel<<<bl, 256, 0, s>>>(x, n, out);
    return cudaGetLastError();
}

}  // namespace skg
