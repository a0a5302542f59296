// skg_tracer.cu -- the wavefront photon-packet tracer.
//
// One phase (stellar emission, dust self-absorption or dust emission) of a batch of wavelengths of
// one or more simulations replaces Parallel::call(this, &dostellaremissionchunk, Nlambda, Nchunks)
// (MonteCarloSimulation.cpp:241-295) and the two dust chunk bodies
// (PanMonteCarloSimulation.cpp:191-346).  The life cycle of a packet,
//
//   launch -> peel-off (emission) -> path: absorption, escape fraction, termination test, forced
//   interaction point -> propagate -> peel-off (scattering) -> scatter -> path -> ...
//
// is cut at its traversals.  The packets in flight sit in a pool of 128-byte records.  Each wave
// runs these kernels:
//   launch_kernel   one thread per packet at its interaction point, then per free record: moves the
//                   packet there and scatters it, or launches a new packet; then puts the packet's next
//                   traversals on the wave's lists (one peel-off job per direction group, one path job);
//   order_kernel    (with its bin kernels, on large waves) the jobs in spatial order;
//   trav_kernel     persistent; each lane takes jobs one after another and walks them, in an
//                   instantiation per kind of walk:
//                   optical depth towards an observer (DustSystem::opticaldepth,
//                   DustSystem.cpp:960-976) or along a path without absorption;
//                   path with absorption: streams kappa*rho*ds into the FP64 cumulative optical depth
//                   and the per-cell tallies (simulateescapeandabsorption, :432-509);
//                   re-walk of a path to the segment where the cumulative optical depth passes the
//                   interaction optical depth, interpolating inside it (DustGridPath::pathlength,
//                   DustGridPath.cpp:162-173);
//   end_kernel      between the walks and the re-walks: per path the escape fraction, the termination
//                   test and the sampling of the interaction optical depth (simulatepropagation, :513-531),
//                   with the next wave's lists of interacting packets and free records; per peel-off the
//                   instruments' tallies.
// The traversal kernels hold nothing but the walk: 64 or 80 registers, with at most 84 bytes of spills (FP64
// paths on trees; a single simulation's FP32 optical depths on octant records 56, on Voronoi and rope records
// none).  What happens to a packet between its walks runs once per packet per wave in kernels of its own.
// Instruments seen from the same direction share one peel-off traversal (identical optical depth; the
// reference recomputes it per instrument).
#include "skg_scene.cuh"
#include "skg_internal.h"
#include "skg_wave.h"
#include <cstring>
#include <type_traits>

#include <chrono>
#include <cstdlib>
#include <map>
#include <mutex>
#include <thread>
#include <tuple>

namespace skg {

#ifndef SKG_TRAV_MIN_BLOCKS
#define SKG_TRAV_MIN_BLOCKS 4
#endif
// The walks of a wave run in kernels of their own (TravMode below): each holds the registers of its
// own state alone, and the path's long end (end_kernel) holds none of them.  Octree disk, 2*10^7
// packets: traversal pass 179.6 ms against 209.8 with the end of the path and the re-walk inside the
// path-job kernel (220 bytes of spills at 64 registers); fit-variant batch 46.2 against 53.5 ms.
// blocks per SM of the path and re-walk kernels: 3 (80 registers; FP32 spills at most 56 bytes) against 4 (64,
// spilling 64-112 bytes): traversal pass of the k-d tree disk with absorption 21.3 against 22.8 ms, Cartesian
// disk with absorption 6.75 against 7.35, re-walks of the octree disk 1.4 ms of 157 less
#ifndef SKG_PATH_MIN_BLOCKS
#define SKG_PATH_MIN_BLOCKS 3
#endif
// programmatic dependent launch of the peel-off-job kernel after the path-job kernel
#ifndef SKG_PDL
#define SKG_PDL 1
#endif
// a lane whose job ended takes the next one when this many lanes of its warp (or all of them) wait for
// one.  With the job records staged by the warp a start costs little: 4, 8 and 12 lanes take the octree
// disk's traversal pass 166.7, 162.3 and 161.5 ms (2*10^7 packets), the fit-variant batch 43.8, 43.3
// and 43.8 ms
#ifndef SKG_REFILL_LANES
#define SKG_REFILL_LANES 8
#endif
// checkpoints of a path's walk (FP32 steppers that can resume): every SKG_CKPT_STRIDE cell steps,
// up to SKG_CKPT_N per packet record, the walk stores its state with the optical depth and path
// length so far; the re-walk to the interaction point then starts at the last checkpoint below the
// interaction optical depth (at most one stride of cell steps) instead of at the path's start
#ifndef SKG_CKPT
#define SKG_CKPT 1
#endif
// cell steps a lane takes per pass of the traversal loop (the warp's refill vote runs once per
// pass): optical-depth and re-walk kernels, path kernel.  2*10^7 packets of the octree disk, ms per pass
// at 5 and 4, 8 and 6, 12 and 8, 16 and 12: 185.3, 180.8, 178.1, 177.9; fit-variant batch 26.4, 25.9, 26.0,
// 26.1 (device); k-d tree disk with absorption 25.4, 24.9, 24.6, 24.5; Voronoi disk 132.7, 132.2, 132.6, 131.2
#ifndef SKG_INNER_STEPS
#define SKG_INNER_STEPS 12
#endif
#ifndef SKG_INNER_PATH
#define SKG_INNER_PATH 8
#endif
#ifndef SKG_CKPT_N
#define SKG_CKPT_N 32
#endif
#ifndef SKG_CKPT_STRIDE
#define SKG_CKPT_STRIDE 16
#endif

// phases of at most this many packets (Cartesian, other grids) run in the tail pass alone: with a few
// lanes of every warp busy a wave lasts as long as its longest walk, about 100 us each on a small Cartesian grid, and a
// phase takes some twenty of them.  Waves against the tail pass alone, ms per phase: 40x40x20 Cartesian
// grid 10^4 packets 1.76 / 1.00, 2*10^4 1.83 / 1.49, 4*10^4 1.98 / 2.23; 100x100x50 2*10^4 2.40 / 2.12, 4*10^4 2.77 /
// 3.48; octree with four observers 4*10^3 1.52 / 1.00, 10^4 1.59 / 1.70; 10^6-leaf k-d tree 10^4 2.97 / 2.96;
// Voronoi, 2*10^4 cells, 4*10^3 5.08 / 3.48, 10^4 5.61 / 5.54; 10^6 cells 4*10^3 22.0 / 16.3, 10^4 24.1 / 24.9
#ifndef SKG_TAIL_ONLY_CART
#define SKG_TAIL_ONLY_CART 20000
#endif
#ifndef SKG_TAIL_ONLY
#define SKG_TAIL_ONLY (1 << 13)
#endif

enum Cnt : int { C_PACKETS = 0, C_STEPS, C_TRAV, C_SCATT, C_PEEL, C_ABS, C_PIX, C_NBR, C_FB, C_ERR, C_N };

template<typename R> SKG_D double rho_load(const DevScene& S, size_t i);
template<> SKG_D double rho_load<double>(const DevScene& S, size_t i) { return __ldg(S.rho + i); }
template<> SKG_D double rho_load<float>(const DevScene& S, size_t i) { return (double)__ldg(S.rhof + i); }

// KappaRho call-back (DustSystem.cpp:459-485)
template<typename R> SKG_D double kappa_rho(const DevScene& S, int m, int ell) {
    if (m < 0) return 0.0;
    if (S.ncomp == 1) return S.kext[ell] * rho_load<R>(S, (size_t)m);
    double r = 0;
    for (int h = 0; h < S.ncomp; h++) r += S.kext[h * S.nlambda + ell] * rho_load<R>(S, (size_t)h * S.ncells + m);
    return r;
}

// Does the stepper carry the density of the step's cell in its leaf record (a data member rho),
// or not (a static constant rho = -1)?
template<typename St> struct EmbeddedRho {
    static constexpr bool value = !std::is_same<decltype(&St::rho), const float*>::value;
};

// kappa*rho of a cell step.  One dust component: kappa_ext of the job's wavelength is held by the
// job (kext1 >= 0) and multiplied in FP32 with the density embedded in the leaf record (tree
// walks), or, in the FP32 walks without records (Cartesian, Voronoi), with the FP32 density table,
// instead of reading the scene's tables every step; the FP64 walks keep the FP64 product of
// KappaRho.  Resolved at compile time per stepper: a run-time choice between the two made the
// lattice walk load the table every step as well (octree traversal pass 7819 against 7212 ms).
template<typename R, typename St>
SKG_D double step_kr(const DevScene& S, const St& st, float kext1, int m, int ell) {
    if constexpr (sizeof(R) == 4 && !EmbeddedRho<St>::value) {
        if (kext1 >= 0.f) return (double)(kext1 * __ldg(S.rhof + m));
        return kappa_rho<R>(S, m, ell);
    } else {
        return (kext1 >= 0.f && st.rho >= 0.f) ? (double)(kext1 * st.rho) : kappa_rho<R>(S, m, ell);
    }
}

// Optical depth of a cell step.  SKG_DTAU32: one dust component on an FP32 walk forms the step's
// kappa*rho*ds in FP32 (the geometry's precision) before the FP64 sum (traversal pass of a phase,
// octree disk 1387 against 1385 ms, k-d tree disk 1745 against 1744 ms: off).
#ifndef SKG_DTAU32
#define SKG_DTAU32 0
#endif
template<typename R, typename St>
SKG_D double step_dtau(const DevScene& S, const St& st, float kext1, int m, int ell, R ds) {
#if SKG_DTAU32
    if constexpr (sizeof(R) == 4) {
        if (kext1 >= 0.f) {
            float r;
            if constexpr (EmbeddedRho<St>::value) r = st.rho; else r = __ldg(S.rhof + m);
            return (double)(kext1 * r * ds);
        }
    }
#endif
    return step_kr<R>(S, st, kext1, m, ell) * (double)ds;
}

// Instrument::detect for the members of one direction group after the shared traversal
// (SEDInstrument.cpp:32-42, FrameInstrument.cpp:33-47, SimpleInstrument.cpp:35-49,
// FullInstrument.cpp:109-177), every tally an atomic.  Returns the number of tally updates.  (detect_peels has the
// same rules for a launch of one simulation, with its SED bins summed per block: a change of one is a change of both.)
// Inlined: as a call it kept a 240-byte stack frame (972 bytes of spill loads per thread at 64 registers against
// 52), and the detections of a 10^7-packet octree phase took 16.1 against 14.3 ms.
#ifndef SKG_DETECT_INLINE
#define SKG_DETECT_INLINE 1
#endif
// frame pixel tallies: lanes of a warp that add to the same pixel sum their values over the warp
// first and one of them adds (1), or every lane adds its own value (0).  Octree disk, 5*10^8
// packets: phase 7870 ms with the aggregation against 7850-7930 ms without, detections 652 against
// 632-640 ms -- lanes of a warp rarely hit one pixel (their packets sit anywhere in the galaxy),
// so the match costs more than the atomics it saves; off by default.
#ifndef SKG_WARP_AGG
#define SKG_WARP_AGG 0
#endif
SKG_D void frame_add(double* addr, double v) {
#if SKG_WARP_AGG
    const unsigned act = __activemask();
    const unsigned peers = __match_any_sync(act, (unsigned long long)addr);
    if (peers & (peers - 1)) {
        double s = 0;
        for (unsigned m = peers; m; m &= m - 1) s += __shfl_sync(peers, v, __ffs(m) - 1);
        v = s;
    }
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(addr, v);
#else
    atomicAdd(addr, v);
#endif
}

#if SKG_DETECT_INLINE
__device__ __forceinline__
#else
__device__ __noinline__
#endif
int detect_group(const DevScene& S, int grp, int ell, double Lpeel, double tau,
                                         int nscatt_peel, bool stellar, int comp, double x, double y, double z) {
    double Lextf = Lpeel * exp(-tau);
    const int nl = S.nlambda;
    int adds = 0;
    for (int q = S.group_start[grp]; q < S.group_start[grp + 1]; q++) {
        const int iq = S.group_instr[q];
        const DevInstr& I = S.instr[iq];
        auto sed_add = [&](int c, double v) {
            atomicAdd(I.sed + (size_t)c * nl + ell, v);
            adds++;
        };
        int l = (I.type == SKG_INSTR_SED) ? -1 : pixel_on_detector(I, x, y, z);
        size_t fp = (size_t)I.nxp * I.nyp;
        if (I.type == SKG_INSTR_FRAME) {
            if (l >= 0) {
                frame_add(I.cube + (size_t)ell * fp + l, Lextf); adds++;
                // the frame of the packet's stellar component (component 1 + comp)
                if (I.ncomp > 1 && comp >= 0) { frame_add(I.cube + ((size_t)(1 + comp) * nl + ell) * fp + l, Lextf); adds++; }
            }
        } else if (I.type == SKG_INSTR_SED) {
            sed_add(0, Lextf);
        } else if (I.type == SKG_INSTR_SIMPLE) {
            sed_add(0, Lextf);
            if (l >= 0) { atomicAdd(I.cube + (size_t)ell * fp + l, Lextf); adds++; }
        } else {
            auto add = [&](int c, double v) {
                sed_add(c, v);
                if (l >= 0) { atomicAdd(I.cube + ((size_t)c * nl + ell) * fp + l, v); adds++; }
            };
            add(SKG_FULL_TOT, Lextf);
            if (stellar) {
                if (nscatt_peel == 0) { add(SKG_FULL_TRA, Lpeel); if (S.ncomp) add(SKG_FULL_STRDIR, Lextf); }
                else {
                    add(SKG_FULL_STRSCA, Lextf);
                    if (nscatt_peel <= I.nscatt_levels) add(SKG_FULL_NBASE + nscatt_peel - 1, Lextf);
                }
            } else {
                if (nscatt_peel == 0) add(SKG_FULL_DUSDIR, Lextf); else add(SKG_FULL_DUSSCA, Lextf);
            }
        }
    }
    return adds;
}

// Packet flags: bit 0 stellar origin, bit 1 the pending peel-offs follow a scattering, bits 8-15
// the launching stellar component + 1 (0: a dust-emission packet).
SKG_D int pk_comp(const Packet& K) { return ((K.flags >> 8) & 0xff) - 1; }

// Does the group need a traversal?  Frame-only groups skip it when the packet projects off every
// frame (FrameInstrument.cpp:36-37).
SKG_D bool group_needs_traversal(const DevScene& S, int grp, double x, double y, double z) {
    if (!S.group_frame_only[grp]) return true;
    for (int q = S.group_start[grp]; q < S.group_start[grp + 1]; q++)
        if (pixel_on_detector(S.instr[S.group_instr[q]], x, y, z) >= 0) return true;
    return false;
}

struct Launched { double x, y, z, kx, ky, kz, L, Lth; int ok; int stellar; int comp; };
SKG_D int pk_flags(const Launched& o) { return (o.stellar ? 1 : 0) | ((o.comp + 1) << 8); }

// Packet launch: StellarSystem::launch (StellarSystem.cpp:116-158) with the geometry samplers
// (GeometricStellarComp.cpp:75-81), or a dust-emission launch from the cell luminosity CDF
// (PanMonteCarloSimulation.cpp:216-224 self-absorption, :301-323 emission with bias).
__device__ __noinline__ Launched launch_packet(const DevGrid& g, const DevScene& S, int phase, int ell,
                                               uint64_t Npp_total, Philox& rng) {
    Launched o;
    o.ok = 0;
    o.comp = -1;
    const int nl = S.nlambda;
    V3<double> pos, dir;
    if (phase == SKG_PHASE_STELLAR) {
        double Lpp = S.Lv[ell] / (double)Npp_total;
        if (!(Lpp > 0)) return o;
        o.Lth = Lpp / S.min_weight_reduction;
        int N = S.nstellar, h = 0;
        double Lw = Lpp;
        if (N > 1) {
            double eb = S.emission_bias;
            double X = rng.uniform();
            if (X < eb) h = max(0, min(N - 1, (int)(N * X / eb)));
            else h = dlocate_clip(S.Xvv + (size_t)ell * (N + 1), N + 1, (X - eb) / (1.0 - eb));
            double Lh = S.starL[h * nl + ell];
            if (!(Lh > 0)) return o;                         // launched with zero luminosity
            Lw = Lpp * (1.0 / (1.0 - eb + eb * (S.Lv[ell] / N) / Lh));
        }
        pos = geom_position(S.stellar[h], rng);
        dir = iso_direction(rng);
        o.L = Lw; o.stellar = 1; o.comp = h;
    } else {
        double Ltot = S.emit_Ltot[ell];
        if (!(Ltot > 0)) return o;
        double Lem = Ltot / (double)Npp_total;
        o.Lth = Lem / S.min_weight_reduction;
        const int nc = S.ncells;
        const double* cdf = S.emit_cdf + (size_t)ell * (nc + 1);
        double X = rng.uniform(), weight = 1.0;
        int m;
        if (phase == SKG_PHASE_DUST_SELFABS) m = dlocate_clip(cdf, nc + 1, X);
        else {
            double xi = S.dust_emission_bias;
            if (X < xi) m = max(0, min(nc - 1, (int)(nc * X / xi)));
            else m = dlocate_clip(cdf, nc + 1, (X - xi) / (1 - xi));
            weight = 1.0 / (1 - xi + xi * (Ltot / nc) / S.emit_Lv[(size_t)ell * nc + m]);
        }
        o.L = Lem * weight;
        if (!(o.L > 0)) return o;
        pos = random_position_in_cell(g, m, rng);
        dir = iso_direction(rng);
        o.stellar = 0;
    }
    o.x = pos.x; o.y = pos.y; o.z = pos.z; o.kx = dir.x; o.ky = dir.y; o.kz = dir.z;
    o.ok = 1;
    return o;
}

// Peel-off weight toward a direction: the Henyey-Greenstein phase function value
// (DustMix.cpp:648-654), weighted by kappa_sca*rho over the components (:319-331).  A negative
// value aborts the peel-off.
__device__ __noinline__ double peel_weight(const DevScene& S, int ell, int cell, double kx, double ky, double kz,
                                           double gx_, double gy_, double gz_) {
    const int nl = S.nlambda;
    double cosalpha = kx * gx_ + ky * gy_ + kz * gz_;
    if (S.ncomp == 1) {
        double gg = S.asym[ell];
        double t = 1.0 + gg * gg - 2 * gg * cosalpha;
        return (1.0 - gg) * (1.0 + gg) / sqrt(t * t * t);
    }
    double sum = 0, acc = 0;
    for (int h = 0; h < S.ncomp; h++) {
        double wv = (cell >= 0) ? S.ksca[h * nl + ell] * S.rho[(size_t)h * S.ncells + cell] : 0.0;
        double gg = S.asym[h * nl + ell];
        double t = 1.0 + gg * gg - 2 * gg * cosalpha;
        acc += wv * (1.0 - gg) * (1.0 + gg) / sqrt(t * t * t);
        sum += wv;
    }
    return (sum > 0) ? acc / sum : -1.0;
}

// Forced interaction optical depth and weight: MonteCarloSimulation::simulatepropagation
// (:513-531) with Random::exponcutoff (Random.cpp:163-176).  Returns tau; L is reweighted.
#ifndef SKG_SAMPLE_INLINE
#define SKG_SAMPLE_INLINE 0
#endif
#if SKG_SAMPLE_INLINE
SKG_D
#else
__device__ __noinline__
#endif
double sample_interaction(double xi, double taupath, double& L, Philox& rng) {
    auto expcut = [&](double xmax) -> double {
        if (xmax < 1e-10) return rng.uniform() * xmax;
        double x;
        int guard = 0;
        do { x = -log1p(-rng.uniform() * (-expm1(-xmax))); } while (x > xmax && ++guard < 64);
        return fmin(x, xmax);
    };
    if (xi == 0.0) return expcut(taupath);
    double X = rng.uniform();
    double ti = (X < xi) ? rng.uniform() * taupath : expcut(taupath);
    double p = -exp(-ti) / expm1(-taupath);
    double q = (1.0 - xi) * p + xi / taupath;
    L *= p / q;
    return ti;
}

// New direction: DustSystem::randomMixForPosition (DustSystem.cpp:855-869) and the
// Henyey-Greenstein sampling of DustMix::scatteringDirectionAndPolarization (DustMix.cpp:595-602).
__device__ __noinline__ V3<double> scatter_direction(const DevScene& S, int ell, int cell, V3<double> k, Philox& rng) {
    const int nl = S.nlambda;
    int h = 0;
    if (S.ncomp > 1 && cell >= 0) {
        double tot = 0, pv[MAX_COMP];
        for (int c = 0; c < S.ncomp; c++) { pv[c] = S.ksca[c * nl + ell] * S.rho[(size_t)c * S.ncells + cell]; tot += pv[c]; }
        double X = rng.uniform(), acc = 0;
        for (h = 0; h < S.ncomp - 1; h++) { acc += pv[h] / tot; if (X < acc) break; }
    }
    double gg = S.asym[h * nl + ell];
    if (fabs(gg) < 1e-6) return iso_direction(rng);
    double f = ((1.0 - gg) * (1.0 + gg)) / (1.0 - gg + 2.0 * gg * rng.uniform());
    double costheta = (1.0 + gg * gg - f * f) / (2.0 * gg);
    return rotate_direction(k, costheta, rng);
}

// finds the work item of global packet p (items sorted by begin; few items)
SKG_D int find_item(const WorkItem* items, int n, uint64_t p) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (items[mid].begin <= p) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------------------------
// launch pass and detections

// Bins of the walk order: the octant of a path job's direction or the group (mod 8) of a peel-off
// job, then the Morton cell of its start on a division of the grid's box.
SKG_D unsigned bin_coord(float u, int bits) {       // u: -1..1 across the box
    const int n = 1 << bits;
    return (unsigned)min(n - 1, max(0, (int)((0.5f * u + 0.5f) * n)));
}
SKG_D unsigned spread3(unsigned v) {                // up to 10 bits, two zeros between
    v = (v | v << 16) & 0x030000FFu; v = (v | v << 8) & 0x0300F00Fu;
    v = (v | v << 4) & 0x030C30C3u; return (v | v << 2) & 0x09249249u;
}
SKG_D unsigned box_bin(float u, float v, float w) {
    const unsigned i = bin_coord(u, BIN_BITS_XY), j = bin_coord(v, BIN_BITS_XY), k = bin_coord(w, BIN_BITS_Z);
    constexpr int D = BIN_BITS_XY - BIN_BITS_Z;     // the finer bits of x and y last
    return (spread3(i >> D) | spread3(j >> D) << 1 | spread3(k) << 2) << (2 * D) | (i & ((1 << D) - 1)) << D | (j & ((1 << D) - 1));
}
SKG_D unsigned path_bin(const DevGrid& g, float x, float y, float z, float kx, float ky, float kz) {
    const unsigned oct = (kx < 0.f ? 1u : 0u) | (ky < 0.f ? 2u : 0u) | (kz < 0.f ? 4u : 0u);
    return oct << (2 * BIN_BITS_XY + BIN_BITS_Z) |
           box_bin((x - g.bmid[0]) * g.bscale[0], (y - g.bmid[1]) * g.bscale[1], (z - g.bmid[2]) * g.bscale[2]);
}
SKG_D unsigned peel_bin(const DevGrid& g, int grp, float x, float y, float z) {
    return (unsigned)(grp & 7) << (2 * BIN_BITS_XY + BIN_BITS_Z) |
           box_bin((x - g.bmid[0]) * g.bscale[0], (y - g.bmid[1]) * g.bscale[1], (z - g.bmid[2]) * g.bscale[2]);
}

// The direction groups that get a peel-off traversal from (x, y, z), as a bit mask
// (MonteCarloSimulation.cpp:299-357): emission peel-offs carry weight 1, scattering peel-offs the
// phase-function value, and a negative value ends the list (the reference aborts the peel-off; it
// takes several dust components).
SKG_D unsigned peel_groups(const DevScene& S, int ell, bool scat, int cell, double kx, double ky, double kz, double x,
                           double y, double z) {
    unsigned need = 0;
    for (int g = 0; g < S.ngroups; g++) {
        if (scat && S.ncomp != 1 && peel_weight(S, ell, cell, kx, ky, kz, S.gkx[g], S.gky[g], S.gkz[g]) < 0) break;
        if (group_needs_traversal(S, g, x, y, z)) need |= 1u << g;
    }
    return need;
}

constexpr int SED_PRIV = 1024;          // SED bins a block keeps privately (8 KB)

// A packet at its interaction point: propagate, count its scattering peel-offs, scatter
// (simulatepropagation :513-531, peeloffscattering :313-357, simulatescattering :535-543).
template<typename R>
SKG_D void scatter_packet(const RunParams& P, int phase, bool peel_on, Packet& K, int& state, unsigned& need,
                          double& kx0, double& ky0, double& kz0) {
    const WorkItem& It = P.items[K.item];
    const DevScene& S = *P.scenes[It.slot];
    const R si = (R)K.s_int;                        // PhotonPackage::propagate
    K.x = (double)((R)K.x + si * (R)K.kx);
    K.y = (double)((R)K.y + si * (R)K.ky);
    K.z = (double)((R)K.z + si * (R)K.kz);
    // the interaction point lies in the cell of its segment (verified by the stepper)
    if (K.s_int > 0) K.pos_cell = (K.int_cell >= 0) ? K.int_cell : -2;
    kx0 = K.kx; ky0 = K.ky; kz0 = K.kz;
    if (peel_on) {
        need = peel_groups(S, K.ell, true, K.int_cell, kx0, ky0, kz0, K.x, K.y, K.z);
    }
    Philox rng;
    rng.init(It.seed, K.id, (uint32_t)K.ell | ((uint32_t)phase << 24));
    rng.c0 = K.rngc;
    const V3<double> kn = scatter_direction(S, K.ell, K.int_cell, mk3(K.kx, K.ky, K.kz), rng);
    K.rngc = rng.c0;
    K.kx = (double)(R)kn.x; K.ky = (double)(R)kn.y; K.kz = (double)(R)kn.z;
    K.nscatt++;
    state = PK_WAIT;
}

// Free records take new packets (all lanes of the warp call this; `need` marks the lanes whose
// record is free): one work-counter atomic per warp; a launch with zero luminosity takes the next
// packet; a record finds none once the work counter is past the batch's packets.
template<typename R>
SKG_D void take_packets(const RunParams& P, const BatchHeader& H, int phase, bool peel_on, int lane, bool need,
                        Packet& K, int& state, unsigned& groups, unsigned& launched) {
    const unsigned FULL = 0xffffffffu;
    while (__any_sync(FULL, need)) {
        const unsigned want = __ballot_sync(FULL, need);
        const int leader = __ffs(want) - 1;
        unsigned long long base = 0;
        if (lane == leader) base = atomicAdd(P.work, (unsigned long long)__popc(want));
        base = __shfl_sync(FULL, base, leader);
        if (need) {
            const uint64_t gp = base + __popc(want & ((1u << lane) - 1));
            if (gp >= H.total) {
                state = PK_DONE; need = false;
            } else {
                const int it = find_item(P.items, H.nitems, gp);
                const WorkItem It = P.items[it];
                const uint64_t q = gp - It.begin;
                const int ei = (int)(q / It.count);
                const uint64_t ip = It.first + (q - (uint64_t)ei * It.count);
                const int ell = P.ells[It.ell0 + ei];
                Philox rng;
                rng.init(It.seed, ip, (uint32_t)ell | ((uint32_t)phase << 24));
                launched++;
                const DevScene& S = *P.scenes[It.slot];
                const Launched o = launch_packet(P.grids[It.slot], S, phase, ell, It.npp_total, rng);
                if (o.ok) {
                    K.x = (double)(R)o.x; K.y = (double)(R)o.y; K.z = (double)(R)o.z;
                    K.kx = (double)(R)o.kx; K.ky = (double)(R)o.ky; K.kz = (double)(R)o.kz;
                    K.L = o.L; K.Lth = o.Lth; K.s_int = 0;
                    K.id = ip; K.item = it; K.ell = ell; K.nscatt = 0;
                    K.pos_cell = -2; K.int_cell = -1; K.rngc = rng.c0;
                    K.flags = pk_flags(o);
                    groups = peel_on ? peel_groups(S, ell, false, -1, 0, 0, 0, K.x, K.y, K.z) : 0;
                    state = S.ncomp > 0 ? PK_WAIT : PK_TERM;    // without dust the life cycle ends here
                    need = false;
                }
            }
        }
    }
}

// Places for every thread's n[i] entries behind the counters at[i] (all threads of a block of 256
// call this, as often as one another): one atomic per block and counter, where one per warp made
// the launches of a wave of 2^21 records wait on a few words of L2.
template<int N> struct BlockPlaces { unsigned warp[2][N][8], base[2][N]; int turn; };
template<int N>
SKG_D void reserve_places(BlockPlaces<N>& sh, int& turn, const unsigned (&n)[N], unsigned* const (&at)[N], unsigned (&place)[N]) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = turn;
    turn ^= 1;                        // (a warp is never two calls ahead of another)
    unsigned inc[N];
    for (int i = 0; i < N; i++) {
        inc[i] = n[i];
        for (int d = 1; d < 32; d <<= 1) { const unsigned v = __shfl_up_sync(FULL, inc[i], d); if (lane >= d) inc[i] += v; }
        if (lane == 31) sh.warp[t][i][warp] = inc[i];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        unsigned sum = 0;
        for (int w = 0; w < 8; w++) { const unsigned v = sh.warp[t][threadIdx.x][w]; sh.warp[t][threadIdx.x][w] = sum; sum += v; }
        unsigned* p = at[0];
        for (int i = 1; i < N; i++) if ((int)threadIdx.x == i) p = at[i];
        sh.base[t][threadIdx.x] = sum ? atomicAdd(p, sum) : 0;
    }
    __syncthreads();
    for (int i = 0; i < N; i++) place[i] = sh.base[t][i] + sh.warp[t][i][warp] + inc[i] - n[i];
}

// Writes a packet's jobs at their places: its path job (path >= 0), its peel-off jobs from j0 on.
SKG_D void write_jobs(const WaveParams& W, int p, const Packet& K, unsigned need, bool path, bool scat, double kx0,
                      double ky0, double kz0, unsigned jm, unsigned j0) {
    const int slot = W.R.items[K.item].slot;
    const DevScene& S = *W.R.scenes[slot];
    for (unsigned m = need; m; m &= m - 1, j0++) {
        const int g = __ffs(m) - 1;
        const double w = scat ? peel_weight(S, K.ell, K.int_cell, kx0, ky0, kz0, S.gkx[g], S.gky[g], S.gkz[g]) : 1.0;
        W.jobs[j0] = make_int2(p, g);
        W.jL[j0] = K.L * w;
        if (W.hist) {
            const unsigned b = peel_bin(W.R.grids[slot], g, (float)K.x, (float)K.y, (float)K.z);
            W.jkey[j0] = make_uint2(b, atomicAdd(W.hist + JOB_BINS + b, 1u));
        }
    }
    if (path) {
        W.jobs[jm] = make_int2(p, JOB_MAIN);
        if (W.hist) {
            const unsigned b = path_bin(W.R.grids[slot], (float)K.x, (float)K.y, (float)K.z, (float)K.kx, (float)K.ky,
                                        (float)K.kz);
            W.jkey[jm] = make_uint2(b, atomicAdd(W.hist + b, 1u));
        }
    }
}

// Scatter-and-launch pass: one thread per packet at its interaction point (propagation, scattering
// peel-offs, scattering), then one per free record (StellarSystem::launch and the samplers, or the
// dust-emission launch), every lane of a warp doing the same work.  The packets' jobs go on the
// wave's lists: path jobs from index 0, a packet's peel-off jobs together from index npool on.  A free record
// that finds no packet is done.
// (3 blocks per SM, 80 registers: launch pass of the octree disk, 10^7 packets, 8.7 ms at 2 blocks and 120
// registers, 7.8 at 3; 4 no faster)
template<typename R>
__global__ void __launch_bounds__(256, 3) launch_kernel(const WaveParams W) {
    __shared__ BlockPlaces<3> sh;
    const RunParams& P = W.R;
    const BatchHeader H = *P.hdr;
    const int phase = H.phase;
    const bool peel_on = phase != SKG_PHASE_DUST_SELFABS;
    const int lane = threadIdx.x & 31;
    int turn = 0;
    unsigned c_scatt = 0, c_packets = 0;
    unsigned* const at[3] = {W.jcount + J_PATH, W.jcount + J_PEEL, W.jnext + J_FREE};
    const unsigned nint = W.wave ? W.jcount[J_INT] : 0;
    for (unsigned b0 = blockIdx.x * blockDim.x; b0 < nint; b0 += gridDim.x * blockDim.x) {
        const unsigned i = b0 + threadIdx.x;
        const bool mine = i < nint;
        const int p = mine ? W.intlist[i] : 0;
        Packet K;
        int state = PK_DONE;
        unsigned need = 0;
        double kx0 = 0, ky0 = 0, kz0 = 0;
        if (mine) {
            K = W.pk[p];
            scatter_packet<R>(P, phase, peel_on, K, state, need, kx0, ky0, kz0);
            c_scatt++;
        }
        const unsigned n[3] = {mine ? 1u : 0u, (unsigned)__popc(need), 0u};
        unsigned place[3];
        reserve_places(sh, turn, n, at, place);
        if (mine) {
            write_jobs(W, p, K, need, true, true, kx0, ky0, kz0, place[0], W.npool + place[1]);
            K.flags |= 2;                         // the pending peel-offs follow a scattering
            K.state = state;
            W.pk[p] = K;
        }
    }
    // (every record is free at first)
    const unsigned nfree = W.wave ? W.jcount[J_FREE] : (unsigned)W.npool;
    for (unsigned b0 = blockIdx.x * blockDim.x; b0 < nfree; b0 += gridDim.x * blockDim.x) {
        const unsigned i = b0 + threadIdx.x;
        const bool mine = i < nfree;
        const int p = !mine ? 0 : W.wave ? W.freelist[i] : (int)i;
        Packet K;
        int state = PK_DONE;
        unsigned need = 0;
        take_packets<R>(P, H, phase, peel_on, lane, mine, K, state, need, c_packets);
        // the start cell once per packet, all lanes together (otherwise each of its walks looks for it)
        if (sizeof(R) == 4 && mine && state != PK_DONE)
            K.pos_cell = start_cell(P.grids[P.items[K.item].slot], (float)K.x, (float)K.y, (float)K.z);
        // (a packet without a path leaves its record free for the next wave)
        const bool path = mine && state == PK_WAIT, ends = mine && state == PK_TERM;
        const unsigned n[3] = {path ? 1u : 0u, (unsigned)__popc(need), ends ? 1u : 0u};
        unsigned place[3];
        reserve_places(sh, turn, n, at, place);
        if (path || ends) write_jobs(W, p, K, need, path, false, 0, 0, 0, place[0], W.npool + place[1]);
        if (ends) W.freenext[place[2]] = p;
        if (mine) {
            K.nck = 0; K.pad[0] = K.pad[1] = K.pad[2] = 0;
            K.state = state;
            if (state == PK_DONE) W.pk[p].state = PK_DONE; else W.pk[p] = K;
        }
    }
    c_scatt = __reduce_add_sync(0xffffffffu, c_scatt);
    c_packets = __reduce_add_sync(0xffffffffu, c_packets);
    if (lane == 0 && c_scatt) atomicAdd(P.counters + C_SCATT, (unsigned long long)c_scatt);
    if (lane == 0 && c_packets) atomicAdd(P.counters + C_PACKETS, (unsigned long long)c_packets);
}

// Adds v to the SED bin key (-1: none) of every lane, the lanes of a bin summed first: the packets of
// a wave share one or two wavelengths, so the lanes' bins are few, and FP64 atomics of a warp on one
// shared-memory word take turns.  All lanes of the warp call this.
SKG_D void sed_add(double* sed, int key, double v) {
    const unsigned FULL = 0xffffffffu;
    unsigned left = __ballot_sync(FULL, key >= 0);
    while (left) {
        const int k0 = __shfl_sync(FULL, key, __ffs(left) - 1);
        double sum = key == k0 ? v : 0.0;
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
        if ((threadIdx.x & 31) == 0) atomicAdd(sed + k0, sum);
        left &= ~__ballot_sync(FULL, key == k0);
    }
}

// Detection: one thread per peel-off job of the wave, right after its walks (Instrument::detect of every
// member of its direction group; detect_group has the rules).  A launch of one simulation tallies its
// SED bins per block and adds them once at the end.  (A pass over all records of the pool in the next wave
// before, which also made the record lists: with the launch pass 35.4 ms a phase of the octree disk, 2*10^7 packets,
// against 26.5; Cartesian disk, 10^6, 2.40 against 1.25; a batch of 24 fit variants 35.1
// against 30.6 ms in all.)
SKG_D void detect_peels(const WaveParams& W, double* s_sed) {
    const RunParams& P = W.R;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int sed_bins = (P.hdr->nslots == 1) ? P.scenes[0]->sed_bins : 0;
    const bool priv = sed_bins > 0 && sed_bins <= SED_PRIV;
    if (priv) for (int t = threadIdx.x; t < sed_bins; t += blockDim.x) s_sed[t] = 0.0;
    __syncthreads();
    unsigned pix = 0, peels = 0;
    const unsigned n = W.jcount[J_PEEL];
    for (unsigned b0 = blockIdx.x * blockDim.x; b0 < n; b0 += gridDim.x * blockDim.x) {
        const unsigned i = b0 + threadIdx.x;
        const bool on = i < n;
        if (!priv) {
            if (on) {
                const unsigned j = W.npool + i;
                const int2 jb = W.jobs[j];
                const Packet& K = W.pk[jb.x];
                const int fl = K.flags;
                pix += detect_group(*P.scenes[P.items[K.item].slot], jb.y, K.ell, W.jL[j], W.jtau[j], (fl & 2) ? K.nscatt : 0,
                                    (fl & 1) != 0, pk_comp(K), K.x, K.y, K.z);
                peels++;
            }
            continue;
        }
        const DevScene& S = *P.scenes[0];
        const int nl = S.nlambda;
        int q0 = 0, q1 = 0, ell = 0, nsp = 0, fl = 0, comp = -1;
        double L = 0, Lext = 0, x = 0, y = 0, z = 0;
        if (on) {
            const unsigned j = W.npool + i;
            const int2 jb = W.jobs[j];
            const Packet& K = W.pk[jb.x];
            q0 = S.group_start[jb.y]; q1 = S.group_start[jb.y + 1];
            fl = K.flags; nsp = (fl & 2) ? K.nscatt : 0; ell = K.ell; comp = pk_comp(K);
            x = K.x; y = K.y; z = K.z;
            L = W.jL[j];
            Lext = L * exp(-W.jtau[j]);
            peels++;
        }
        const int members = __reduce_max_sync(FULL, q1 - q0);
        for (int q = 0; q < members; q++) {
            int key[3] = {-1, -1, -1};
            double v[3] = {0, 0, 0};
            if (q0 + q < q1) {
                const int iq = S.group_instr[q0 + q];
                const DevInstr& I = S.instr[iq];
                const int c0 = S.sed_base[iq] + ell;
                const int l = (I.type == SKG_INSTR_SED) ? -1 : pixel_on_detector(I, x, y, z);
                const size_t fp = (size_t)I.nxp * I.nyp;
                if (I.type != SKG_INSTR_FRAME) { key[0] = c0; v[0] = Lext; pix++; }
                if (l >= 0) { atomicAdd(I.cube + (size_t)ell * fp + l, Lext); pix++; }
                if (I.type == SKG_INSTR_FRAME) {
                    // the frame of the packet's stellar component (component 1 + comp)
                    if (l >= 0 && I.ncomp > 1 && comp >= 0) {
                        atomicAdd(I.cube + ((size_t)(1 + comp) * nl + ell) * fp + l, Lext); pix++;
                    }
                } else if (I.type == SKG_INSTR_FULL) {
                    auto add = [&](int s, int c, double value) {
                        key[s] = c0 + c * nl; v[s] = value; pix++;
                        if (l >= 0) { atomicAdd(I.cube + ((size_t)c * nl + ell) * fp + l, value); pix++; }
                    };
                    if (fl & 1) {
                        if (nsp == 0) { add(1, SKG_FULL_TRA, L); if (S.ncomp) add(2, SKG_FULL_STRDIR, Lext); }
                        else {
                            add(1, SKG_FULL_STRSCA, Lext);
                            if (nsp <= I.nscatt_levels) add(2, SKG_FULL_NBASE + nsp - 1, Lext);
                        }
                    } else {
                        add(1, nsp == 0 ? SKG_FULL_DUSDIR : SKG_FULL_DUSSCA, Lext);
                    }
                }
            }
            __syncwarp();
            for (int s = 0; s < 3; s++) sed_add(s_sed, key[s], v[s]);
        }
    }
    pix = __reduce_add_sync(FULL, pix);
    peels = __reduce_add_sync(FULL, peels);
    if (lane == 0 && pix) atomicAdd(P.counters + C_PIX, (unsigned long long)pix);
    if (lane == 0 && peels) atomicAdd(P.counters + C_PEEL, (unsigned long long)peels);
    if (!priv) return;
    __syncthreads();
    const DevScene& S0 = *P.scenes[0];
    for (int t = threadIdx.x; t < sed_bins; t += blockDim.x) {
        const double v = s_sed[t];
        if (v == 0.0) continue;
        int i = 0;
        while (i + 1 < S0.ninstr && S0.sed_base[i + 1] <= t) i++;
        atomicAdd(S0.instr[i].sed + (t - S0.sed_base[i]), v);
    }
}

// ---------------------------------------------------------------------------------------------
// walk order: a counting sort of the wave's jobs by bin (each job has its rank within its bin from
// the launch pass)

// First place of each bin: the counts of the bins before it among path jobs or among peel-off jobs.
// Blocks of 1024 threads, 8 bins a thread; bin_sums_kernel sums each block's bins first.
constexpr int BIN_BLOCK = 8192;
SKG_D unsigned warp_sum(unsigned v) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
__global__ void __launch_bounds__(1024) bin_sums_kernel(const unsigned* __restrict__ hist, unsigned* sums) {
    __shared__ unsigned ws[32];
    const uint4* h = reinterpret_cast<const uint4*>(hist + (size_t)blockIdx.x * BIN_BLOCK);
    const uint4 a = h[threadIdx.x], b = h[threadIdx.x + 1024];
    const unsigned v = warp_sum(a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned t = warp_sum(ws[threadIdx.x]);
        if (threadIdx.x == 0) sums[blockIdx.x] = t;
    }
}
// Clears the counts as well.
__global__ void __launch_bounds__(1024) bins_kernel(unsigned* hist, unsigned* bin0, const unsigned* __restrict__ sums) {
    __shared__ unsigned ws[32], before;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* h = reinterpret_cast<uint4*>(hist + (size_t)blockIdx.x * BIN_BLOCK) + 2 * threadIdx.x;
    uint4* o = reinterpret_cast<uint4*>(bin0 + (size_t)blockIdx.x * BIN_BLOCK) + 2 * threadIdx.x;
    uint4 c[2];
    unsigned sum = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) { c[i] = h[i]; sum += c[i].x + c[i].y + c[i].z + c[i].w; }
    unsigned inc = sum;
    for (int d = 1; d < 32; d <<= 1) { const unsigned t = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= d) inc += t; }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        constexpr int HALF = JOB_BINS / BIN_BLOCK;
        unsigned v = 0;
        for (int b = blockIdx.x / HALF * HALF + lane; b < (int)blockIdx.x; b += 32) v += sums[b];
        v = warp_sum(v);
        const unsigned t = ws[lane];
        unsigned w = t;
        for (int d = 1; d < 32; d <<= 1) { const unsigned q = __shfl_up_sync(0xffffffffu, w, d); if (lane >= d) w += q; }
        ws[lane] = w - t;
        if (lane == 0) before = v;
    }
    __syncthreads();
    unsigned at = before + ws[warp] + inc - sum;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        uint4 b;
        b.x = at; at += c[i].x; b.y = at; at += c[i].y; b.z = at; at += c[i].z; b.w = at; at += c[i].w;
        o[i] = b;
        h[i] = make_uint4(0, 0, 0, 0);
    }
}

// Writes the jobs in walk order.
__global__ void __launch_bounds__(256) order_kernel(const WaveParams W) {
    const unsigned npath = W.jcount[J_PATH], n = npath + W.jcount[J_PEEL];
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned j = i < npath ? i : W.npool + (i - npath);
        const uint2 k = W.jkey[j];
        const int2 jb = W.jobs[j];
        if (i < npath) W.spath[W.bin0[k.x] + k.y] = jb.x;
        else W.speel[W.bin0[JOB_BINS + k.x] + k.y] = make_uint2((unsigned)jb.x << 4 | (unsigned)jb.y, j);
    }
}

// ---------------------------------------------------------------------------------------------
// traversal pass

// 1 - e^-x for x >= 0, to about one unit in the last place: the Taylor series up to x^10 below 1/16
// (its next term is below 10^-19 of the sum), expm1 above.  A path step's optical depth is small, and the
// series takes ten FP64 operations and no branches.
SKG_D double one_minus_exp(double x) {
    if (x < 0.0625) {
        double p = -1.0 / 3628800;
        p = fma(p, x, 1.0 / 362880);
        p = fma(p, x, -1.0 / 40320);
        p = fma(p, x, 1.0 / 5040);
        p = fma(p, x, -1.0 / 720);
        p = fma(p, x, 1.0 / 120);
        p = fma(p, x, -1.0 / 24);
        p = fma(p, x, 1.0 / 6);
        p = fma(p, x, -0.5);
        p = fma(p, x, 1.0);
        return p * x;
    }
    return -expm1(-x);
}

// Absorption in cell m of a path step: simulateescapeandabsorption (MonteCarloSimulation.cpp:441-462)
// with OligoDustSystem::absorb / PanDustSystem::absorb.  The tables are wavelength-major on the
// device ([ell][m]): a wave carries the packets of one or two wavelengths (packets are handed out
// wavelength by wavelength), so its tallies fall in one slice of the table that stays in L2.
// v1 = L e^-tau on entry (a running product, each step absorbs v1 (1 - e^-dtau)); v2 accumulates L_sca
// with the local albedo when there are several dust components.  Returns 1 when a tally was stored.
template<typename R>
SKG_D int absorb_step(const DevScene& S, int phase, int m, int ell, double dtau, double& v1, double& v2) {
    if (m < 0) return 0;
    const bool store = (phase == SKG_PHASE_STELLAR) ? (S.store_abs != 0) : (phase == SKG_PHASE_DUST_SELFABS);
    double* labs = (phase == SKG_PHASE_STELLAR) ? S.labs_stel : S.labs_dust;
    if (S.ncomp == 1) {
        if (!store) return 0;
        const double Lintm = v1 * one_minus_exp(dtau);
        v1 -= Lintm;
        atomicAdd(labs + (size_t)ell * S.ncells + m, (1.0 - S.albedo[ell]) * Lintm);
        return 1;
    }
    double ksca = 0, kext = 0;
    for (int h = 0; h < S.ncomp; h++) {
        const double rh = rho_load<R>(S, (size_t)h * S.ncells + m);
        ksca += rh * S.ksca[h * S.nlambda + ell]; kext += rh * S.kext[h * S.nlambda + ell];
    }
    const double alb = (kext > 0.0) ? ksca / kext : 0.0;
    const double Lintm = v1 * one_minus_exp(dtau);
    v1 -= Lintm;
    v2 += alb * Lintm;
    if (!store) return 0;
    atomicAdd(labs + (size_t)ell * S.ncells + m, (1.0 - alb) * Lintm);
    return 1;
}

// End of the packet's own path (simulateescapeandabsorption :441-462, the termination test of
// dostellaremissionchunk :283, simulatepropagation :513-531).  Returns 1 when the path must be
// re-walked to tau_int (the packet's luminosity is then already in its record), 0 when the packet
// record is complete, -1 on an error.  Inlined: as a call
// it made the traversal kernel keep a 264-byte stack frame for the call's saved registers (88
// bytes inlined; the traversal pass ran 11 % faster).
SKG_D int after_path(const WaveParams& W, const DevScene& S, int p, int phase, int ell,
                     double taupath, double Lsca, double& L, double& tau_int) {
    Packet& K = W.pk[p];
    if (taupath < 0.0 || isnan(taupath) || isinf(taupath)) {   // DustSystem.cpp:953-955
        atomicOr(W.R.err, ERR_NAN_TAU);
        K.state = PK_TERM;
        return -1;
    }
    if (S.ncomp == 1) L = L * S.albedo[ell] * (-expm1(-taupath));
    else L = Lsca;
    if (L <= 0 || (L <= K.Lth && K.nscatt >= S.min_scatt_events)) { K.state = PK_TERM; return 0; }
    if (K.nscatt >= W.R.max_scatt) {
        atomicOr(W.R.err, ERR_SCATT_BUDGET);
        K.state = PK_TERM;
        return -1;
    }
    if (taupath == 0.0) {                 // no dust ahead: scatter where the packet is
        K.L = L; K.s_int = 0; K.int_cell = K.pos_cell >= 0 ? K.pos_cell : -1; K.state = PK_INTERACT;
        return 0;
    }
    const WorkItem& It = W.R.items[K.item];
    Philox rng;
    rng.init(It.seed, K.id, (uint32_t)ell | ((uint32_t)phase << 24));
    rng.c0 = K.rngc;
    tau_int = sample_interaction(S.xi, taupath, L, rng);
    K.rngc = rng.c0;
    K.L = L;                              // the weight the packet carries to its interaction point
    return 1;
}

// A checkpoint of packet p's path walk (slot i): the stepper's state, then the optical depth and
// the path length walked (from the packet's position) and the step count.
template<class St>
SKG_D void save_ckpt(const WaveParams& W, int p, int i, const St& st, double tau) {
    const Packet& K = W.pk[p];
    const float s = st.walked_from((float)K.x, (float)K.y, (float)K.z);
    float4* c = W.ckpt + ((size_t)p * SKG_CKPT_N + i) * 2;
    c[0] = st.ckpt();
    c[1] = make_float4(__int_as_float(__double2loint(tau)), __int_as_float(__double2hiint(tau)), s,
                       __int_as_float(st.steps));
}

// Resumes the re-walk of packet p's path toward tau_int at its last checkpoint (of nck) whose
// optical depth is at most tau_int: the steps before it would not have reached tau_int.  Returns
// false when there is none (the re-walk starts at the path's start).
template<class St>
SKG_D bool resume_ckpt(const WaveParams& W, const DevGrid& g, int p, int nck, double tau_int, St& st, double& tau,
                       double& s) {
    const float4* c = W.ckpt + (size_t)p * SKG_CKPT_N * 2;
    int lo = -1, hi = nck - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const float4 b = c[2 * mid + 1];
        if (__hiloint2double(__float_as_int(b.y), __float_as_int(b.x)) <= tau_int) lo = mid; else hi = mid - 1;
    }
    if (lo < 0) return false;
    const float4 b = c[2 * lo + 1];
    const Packet& K = W.pk[p];
    st.resume(g, (float)K.x, (float)K.y, (float)K.z, (float)K.kx, (float)K.ky, (float)K.kz, K.pos_cell, c[2 * lo],
              __float_as_int(b.w));
    tau = __hiloint2double(__float_as_int(b.y), __float_as_int(b.x));
    s = (double)b.z;
    return true;
}

// The walks of a wave, each in an instantiation that holds its own state alone:
//   TRAV_PATH    the path jobs of phases that keep absorption or of several dust components
//   TRAV_TAU     jobs that need the optical depth alone: the peel-offs, and the path jobs otherwise
//   TRAV_REWALK  the paths that interact, to the interaction optical depth
enum TravMode : int { TRAV_PATH = 1, TRAV_TAU = 2, TRAV_REWALK = 3 };
// Resident blocks per SM of each instantiation.
template<int MODE, template<typename> class Stepper> struct TravBlocks { static constexpr int value = SKG_TRAV_MIN_BLOCKS; };
template<template<typename> class Stepper> struct TravBlocks<TRAV_PATH, Stepper> { static constexpr int value = SKG_PATH_MIN_BLOCKS; };
template<> struct TravBlocks<TRAV_TAU, VoronoiStepper> { static constexpr int value = 3; };   // 12 planes in flight
template<template<typename> class Stepper> struct TravBlocks<TRAV_REWALK, Stepper> { static constexpr int value = SKG_PATH_MIN_BLOCKS; };

template<typename R, template<typename> class Stepper>
struct HasCkpt { static constexpr bool value = SKG_CKPT && Resumable<Stepper<R>>::value; };

template<typename R, template<typename> class Stepper, int MODE, bool ONE>
__global__ void __launch_bounds__(256, (TravBlocks<MODE, Stepper>::value)) trav_kernel(const WaveParams W) {
    extern __shared__ unsigned char smem_raw[];
    DevGrid* sg = reinterpret_cast<DevGrid*>(smem_raw);
    // the grid of a job's slot: a single-simulation launch (ONE) reads it from the kernel's
    // parameters, whose fields are constant-bank operands; a batch from the block's shared copy,
    // which the compiler reloads after the shared-memory counter atomics of the loop
    auto grid_of = [&](int sl) -> const DevGrid& {
        if constexpr (ONE) return W.g0; else return sg[sl];
    };
    __shared__ const DevScene* s_scene[MAX_SLOTS];
    __shared__ unsigned long long s_cnt[C_N];
    const RunParams& P = W.R;
    const BatchHeader H = *P.hdr;
    for (int i = threadIdx.x; i < C_N; i += blockDim.x) s_cnt[i] = 0;
    for (int i = threadIdx.x; i < H.nslots; i += blockDim.x) { sg[i] = P.grids[i]; s_scene[i] = P.scenes[i]; }
    __syncthreads();
#if SKG_PDL
    // the path-job kernel lets the peel-off-job kernel of the same wave be scheduled now: its blocks
    // become resident as this kernel's blocks run out of jobs and exit, so the two overlap in the
    // tail of this one.  The peel-off kernel reads only what the launch pass wrote (complete before
    // this kernel started); the one word both may touch, a packet's start cell, is written here
    // only from "unknown" to the cell, and either value is a valid hint for the peel-off walk.
    if (MODE == TRAV_PATH) asm volatile("griddepcontrol.launch_dependents;");
#endif
    // the walk's jobs in the wave's list
    const unsigned npath = W.jcount[J_PATH];
    const unsigned job0 = (MODE == TRAV_TAU && !W.path_tau) ? npath : 0;   // (re-walks: listed by the path ends)
    const unsigned njobs = MODE == TRAV_PATH ? npath : MODE == TRAV_TAU ? npath - job0 + W.jcount[J_PEEL] : W.jcount[J_REWALK];
    unsigned* const taken = W.jcount + (MODE == TRAV_PATH ? J_TAKEN_PATH : MODE == TRAV_TAU ? J_TAKEN_TAU : J_TAKEN_REWALK);
    const int phase = H.phase;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int refill_lanes = P.refill > 0 ? P.refill : SKG_REFILL_LANES;
    constexpr bool CKPT = HasCkpt<R, Stepper>::value;
    // A warp takes jobs in chunks of up to 32 and stages their records in shared memory, all lanes
    // loading at once: the chain of dependent loads of a job start (job, packet, tables) is paid once
    // per chunk instead of once per refill, and the lanes walk neighbours in walk order.  A wave with
    // fewer jobs than lanes spreads them over the warps.  Fit-variant batch 39.5 against 46.2 ms,
    // octree disk (2*10^7 packets) traversal pass 162.3 against 171.2 ms.
    __shared__ WalkJob<R> s_job[256];
    WalkJob<R>* const mine = s_job + (threadIdx.x & ~31);
    const unsigned nwarps = gridDim.x * 8;
    const int chunk = (int)min(32u, max(1u, (njobs + nwarps - 1) / nwarps));
    int have = 0, used = 0;           // jobs of the chunk, and those handed to lanes
    bool more = true;                 // the list has jobs left

    int j = -1;                       // where the lane's job leaves its result (-1: no job)
    int p = 0, slot = 0, ell = 0;
    double tau = 0;                   // optical depth walked
    // TRAV_PATH: v1 = L e^-tau (the luminosity that reaches the current cell, kept as a running
    // product), v2 = L_sca (several dust components);
    // TRAV_REWALK: v1 = path length walked, v2 = the interaction optical depth
    double v1 = 0, v2 = 0;
    float kext1 = -1.f;
    unsigned c_steps = 0, c_trav = 0, c_fb = 0, c_abs = 0;
    unsigned long long c_nbr = 0;
    Stepper<R> st;
    int nck = 0;                      // checkpoints of the path walk
    double* labs = nullptr;           // TRAV_PATH: tallies of the job's wavelength (one dust component), if kept
    double kabs = 0;                  // 1 - albedo

    while (true) {
        const unsigned want = __ballot_sync(FULL, j < 0);
        if (want && (__popc(want) >= refill_lanes || want == FULL)) {
            if (used == have && more) {
                unsigned base = 0;
                if (lane == 0) base = atomicAdd(taken, (unsigned)chunk);
                base = __shfl_sync(FULL, base, 0);
                have = base < njobs ? (int)min((unsigned)chunk, njobs - base) : 0;
                used = 0;
                more = have > 0;
                if (lane < have) {
                    WalkJob<R> w;
                    const unsigned i = job0 + base + lane;
                    int grp = JOB_MAIN;
                    if (MODE == TRAV_REWALK) {
                        const int2 r = W.rlist[i];
                        w.p = r.x; w.out = r.y;
                    } else if (MODE == TRAV_PATH || i < npath) {
                        w.p = W.hist ? W.spath[i] : W.jobs[i].x;
                        w.out = (int)i;
                    } else if (W.hist) {
                        const uint2 o = W.speel[i - npath];
                        w.p = (int)(o.x >> 4); grp = (int)(o.x & 15); w.out = (int)o.y;
                    } else {
                        w.out = W.npool + (int)(i - npath);
                        const int2 jb = W.jobs[w.out];
                        w.p = jb.x; grp = jb.y;
                    }
                    const Packet& K = W.pk[w.p];
                    w.ell = K.ell; w.hint = K.pos_cell;
                    w.slot = ONE ? 0 : P.items[K.item].slot;
                    const DevScene& S = *s_scene[w.slot];
                    if (HasGroups<Stepper<R>>::value && MODE == TRAV_TAU) w.slot |= grp << 8;
                    w.kext1 = (S.ncomp == 1) ? (float)S.kext[w.ell] : -1.f;
                    w.x = (R)K.x; w.y = (R)K.y; w.z = (R)K.z;
                    if (MODE != TRAV_TAU || grp == JOB_MAIN) { w.kx = (R)K.kx; w.ky = (R)K.ky; w.kz = (R)K.kz; }
                    else { w.kx = (R)S.gkx[grp]; w.ky = (R)S.gky[grp]; w.kz = (R)S.gkz[grp]; }
                    mine[lane] = w;
                }
                __syncwarp();
            }
            if (used == have) {
                if (want == FULL) break;
            } else {
                const int r = used + __popc(want & ((1u << lane) - 1));
                if (j < 0 && r < have) {
                    const WalkJob<R> w = mine[r];
                    j = w.out; p = w.p; slot = w.slot & 255; ell = w.ell; kext1 = w.kext1;
                    tau = 0;
                    const DevGrid& g = grid_of(slot);
                    if constexpr (HasGroups<Stepper<R>>::value)
                        st.group = (MODE == TRAV_TAU && (w.slot >> 8) != JOB_MAIN && g.gplane) ? w.slot >> 8 : -1;
                    // entry segments outside the grid (m = -1) carry no optical depth: only the
                    // re-walk, which measures length, takes them
                    if (MODE == TRAV_REWALK) {
                        v1 = 0; v2 = W.jtau[j];
                        bool resumed = false;
                        if constexpr (CKPT) resumed = W.ckpt && resume_ckpt(W, g, p, W.pk[p].nck, v2, st, tau, v1);
                        if (!resumed) {
                            st.init(g, w.x, w.y, w.z, w.kx, w.ky, w.kz, w.hint);
                            R d0;
                            while (st.pd.pop(d0)) v1 += (double)d0;
                        }
                    } else {
                        st.init(g, w.x, w.y, w.z, w.kx, w.ky, w.kz, w.hint);
                        nck = 0;
                        if ((MODE == TRAV_PATH || j < (int)npath) && w.hint == -2) W.pk[p].pos_cell = st.cell0;
                        if (MODE == TRAV_PATH) {
                            v1 = W.pk[p].L; v2 = 0;
                            const DevScene& S = *s_scene[slot];
                            labs = nullptr;
                            if (S.ncomp == 1 && (phase == SKG_PHASE_STELLAR ? S.store_abs != 0 : phase == SKG_PHASE_DUST_SELFABS)) {
                                labs = (phase == SKG_PHASE_STELLAR ? S.labs_stel : S.labs_dust) + (size_t)ell * S.ncells;
                                kabs = 1.0 - S.albedo[ell];
                            }
                        }
                    }
                }
                used = min(have, used + __popc(want));
                __syncwarp();
            }
        }

        if (j < 0) continue;            // waiting for enough lanes to refill

        const DevGrid& g = grid_of(slot);
        const DevScene& S = *s_scene[slot];
        // a checkpoint of a path's walk every SKG_CKPT_STRIDE steps
        auto checkpoint = [&](bool path) {
            if constexpr (CKPT) {
                if (path && W.ckpt && nck < SKG_CKPT_N && st.steps >= (nck + 1) * SKG_CKPT_STRIDE && !st.done) {
                    save_ckpt(W, p, nck, st, tau);
                    nck++;
                }
            }
        };
        // cell steps: several of them before the warp looks at refills again.  (Walking
        // four steps ahead and loading their densities together, for the walks whose records do
        // not carry the density, was slower: Cartesian traversal pass 83 against 64 ms, Voronoi
        // peel-off walks 298 against 258 ms; the walk is issue-bound, not waiting on those loads.)
#pragma unroll 1
        for (int is = 0; is < (MODE == TRAV_PATH ? SKG_INNER_PATH : SKG_INNER_STEPS); is++) {
            int m; R ds;
            if (st.walk(g, m, ds)) {
                c_steps++;
                const double dtau = step_dtau<R>(S, st, kext1, m, ell, ds);
                if (MODE == TRAV_TAU) {
                    tau += dtau;
                    if constexpr (CKPT) checkpoint(j < (int)npath);
                } else if (MODE == TRAV_PATH) {
                    if (labs) {
                        const double Lintm = v1 * one_minus_exp(dtau);
                        v1 -= Lintm;
                        atomicAdd(labs + m, kabs * Lintm);
                        c_abs++;
                    } else if (kext1 < 0.f) {
                        c_abs += absorb_step<R>(S, phase, m, ell, dtau, v1, v2);
                    }
                    tau += dtau;
                    if constexpr (CKPT) checkpoint(true);
                } else {
                    const double tn = tau + dtau, sn = v1 + (double)ds;
                    if (tn > v2) {
                        Packet& K = W.pk[p];
                        K.s_int = v1 + ((v2 - tau) / (tn - tau)) * (sn - v1);
                        K.int_cell = m;
                        K.state = PK_INTERACT;
                        c_trav++; c_nbr += st.nscanned(); c_fb += st.fallbacks;
                        j = -1;
                        break;
                    }
                    tau = tn; v1 = sn;
                }
            } else {
                // the traversal reached the edge of the grid
                c_trav++; c_nbr += st.nscanned(); c_fb += st.fallbacks;
                if (st.steps > g.max_steps) { atomicOr(P.err, ERR_STEP_BUDGET); atomicAdd(&s_cnt[C_ERR], 1ull); }
                if (MODE == TRAV_REWALK) {
                    // DustGridPath::pathlength: an optical depth beyond the last segment gives the full length
                    Packet& K = W.pk[p];
                    K.s_int = v1; K.int_cell = -1; K.state = PK_INTERACT;
                } else {
                    W.jtau[j] = tau;
                    if (MODE == TRAV_PATH) W.jL[j] = v2;
                    if (CKPT && (MODE == TRAV_PATH || j < (int)npath)) W.pk[p].nck = nck;
                }
                j = -1;
                break;
            }
        }
    }

    // the counters, once per lane
    atomicAdd(&s_cnt[C_STEPS], (unsigned long long)c_steps);
    atomicAdd(&s_cnt[C_TRAV], (unsigned long long)c_trav);
    atomicAdd(&s_cnt[C_NBR], c_nbr);
    atomicAdd(&s_cnt[C_FB], (unsigned long long)c_fb);
    if (MODE == TRAV_PATH) atomicAdd(&s_cnt[C_ABS], (unsigned long long)c_abs);
    __syncthreads();
    if (threadIdx.x < C_N && s_cnt[threadIdx.x]) atomicAdd(P.counters + threadIdx.x, s_cnt[threadIdx.x]);
#if SKG_PDL
    // the peel-off kernel completes only after the path-job kernel it overlapped (and its writes
    // are visible), so what follows it in the stream sees both
    if (MODE == TRAV_TAU) asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// The ends of the wave's paths, one thread per path job in walk order: escape fraction, termination
// test and interaction optical depth (after_path).  The packets that interact go on the re-walk list
// and on the next wave's interaction list, the records of the others on its free list.
// Outside the walks every lane of a warp does this long FP64 work at once, and the walks need no
// registers for it.
SKG_D void end_paths(const WaveParams& W, BlockPlaces<3>& sh) {
    const RunParams& P = W.R;
    const unsigned n = W.jcount[J_PATH];
    const int phase = P.hdr->phase;
    int turn = 0;
    unsigned* const at[3] = {W.jcount + J_REWALK, W.jnext + J_INT, W.jnext + J_FREE};
    if (blockIdx.x == 0 && threadIdx.x == 0 && n + W.jcount[J_PEEL] > 0) *W.last_busy = (unsigned)W.wave;
    for (unsigned b0 = blockIdx.x * blockDim.x; b0 < n; b0 += gridDim.x * blockDim.x) {
        const unsigned i = b0 + threadIdx.x;
        bool again = false, inter = false;
        int p = 0;
        if (i < n) {
            p = W.hist ? W.spath[i] : W.jobs[i].x;
            const Packet& K = W.pk[p];
            const DevScene& S = *P.scenes[P.items[K.item].slot];
            double L = K.L, tau_int = 0;
            const int rc = after_path(W, S, p, phase, K.ell, W.jtau[i], W.path_tau ? 0.0 : W.jL[i], L, tau_int);
            if (rc < 0) atomicAdd(P.counters + C_ERR, 1ull);
            again = rc == 1;
            inter = again || (rc == 0 && K.state == PK_INTERACT);
            if (again) W.jtau[i] = tau_int;
        }
        const unsigned cnt[3] = {again ? 1u : 0u, inter ? 1u : 0u, i < n && !inter ? 1u : 0u};
        unsigned place[3];
        reserve_places(sh, turn, cnt, at, place);
        if (again) W.rlist[place[0]] = make_int2(p, (int)i);
        if (inter) W.intnext[place[1]] = p;
        else if (i < n) W.freenext[place[2]] = p;
    }
}

// The ends of the paths and the detections of a wave in one launch, after its walks (as two, a batch of
// 24 fit variants 27.3 against 26.4 ms, an octree phase of 2.4*10^5 packets 2.92 against 2.83).
__global__ void __launch_bounds__(256) end_kernel(const WaveParams W) {
    __shared__ BlockPlaces<3> sh;
    __shared__ double s_sed[SED_PRIV];
    end_paths(W, sh);
    detect_peels(W, s_sed);
}

// ---------------------------------------------------------------------------------------------
// tail pass: the end of a phase
//
// When few packets are left in flight, each wave costs about as long as its longest walk while
// most of the device idles, and a packet still needs a wave per event.  The tail pass gives every
// remaining packet a thread that runs the rest of its life at once -- interaction, scattering peel-offs,
// scattering, path and re-walk until it terminates, then further packets while the work counter has any -- with
// the same random streams, samplers and tallies as the waves (device functions shared with their kernels), so a phase gives the same results with or without it, up to the summation order of the
// FP64 tally atomics.

// Optical depth from (x, y, z) toward (kx, ky, kz) to the edge of the grid (DustSystem::opticaldepth,
// DustSystem.cpp:960-976).
template<typename R, template<typename> class Stepper>
SKG_D double tail_tau(const DevGrid& g, const DevScene& S, int ell, R x, R y, R z, R kx, R ky, R kz, int hint,
                      unsigned long long* cnt, unsigned* err) {
    Stepper<R> st;
    st.init(g, x, y, z, kx, ky, kz, hint);
    const float kext1 = (S.ncomp == 1) ? (float)S.kext[ell] : -1.f;
    double tau = 0;
    int m; R ds;
    while (st.walk(g, m, ds)) {
        cnt[C_STEPS]++;
        tau += step_dtau<R>(S, st, kext1, m, ell, ds);
    }
    cnt[C_TRAV]++; cnt[C_NBR] += st.nscanned(); cnt[C_FB] += st.fallbacks;
    if (st.steps > g.max_steps) { atomicOr(err, ERR_STEP_BUDGET); cnt[C_ERR]++; }
    return tau;
}

// The peel-offs of the packet from its position (peeloffemission :299-309, peeloffscattering
// :313-357): one traversal per direction group that needs one, detected at once.  nsp: the
// scattering count the peel-off copy carries (0 for emission).
template<typename R, template<typename> class Stepper>
SKG_D void tail_peel(const DevGrid& g, const DevScene& S, const Packet& K, bool scat, int nsp, double kx0,
                     double ky0, double kz0, unsigned long long* cnt, unsigned* err) {
    for (int grp = 0; grp < S.ngroups; grp++) {
        double w = 1.0;
        if (scat) {
            w = peel_weight(S, K.ell, K.int_cell, kx0, ky0, kz0, S.gkx[grp], S.gky[grp], S.gkz[grp]);
            if (w < 0) break;
        }
        if (!group_needs_traversal(S, grp, K.x, K.y, K.z)) continue;
        const double tau = tail_tau<R, Stepper>(g, S, K.ell, (R)K.x, (R)K.y, (R)K.z, (R)S.gkx[grp], (R)S.gky[grp],
                                                (R)S.gkz[grp], K.pos_cell, cnt, err);
        cnt[C_PEEL]++;
        cnt[C_PIX] += detect_group(S, grp, K.ell, K.L * w, tau, nsp, (K.flags & 1) != 0, pk_comp(K), K.x, K.y, K.z);
    }
}

// The packet's own path and, when it interacts, the re-walk to the interaction point: the path job
// of the traversal pass.  Leaves the record in PK_INTERACT or PK_TERM.
template<typename R, template<typename> class Stepper>
SKG_D void tail_path(const WaveParams& W, const DevGrid& g, const DevScene& S, int p, int phase,
                     unsigned long long* cnt) {
    Packet& K = W.pk[p];
    const int ell = K.ell;
    const float kext1 = (S.ncomp == 1) ? (float)S.kext[ell] : -1.f;
    Stepper<R> st;
    const int hint = K.pos_cell;
    st.init(g, (R)K.x, (R)K.y, (R)K.z, (R)K.kx, (R)K.ky, (R)K.kz, hint);
    if (hint == -2) K.pos_cell = st.cell0;
    double tau = 0, v1 = K.L, v2 = 0;
    constexpr bool CKPT = SKG_CKPT && Resumable<Stepper<R>>::value;
    int nck = 0;                                  // checkpoints, as the traversal pass takes them
    int m; R ds;
    while (st.walk(g, m, ds)) {
        cnt[C_STEPS]++;
        const double dtau = step_dtau<R>(S, st, kext1, m, ell, ds);
        cnt[C_ABS] += absorb_step<R>(S, phase, m, ell, dtau, v1, v2);
        tau += dtau;
        if constexpr (CKPT) {
            if (W.ckpt && nck < SKG_CKPT_N && st.steps >= (nck + 1) * SKG_CKPT_STRIDE && !st.done) {
                save_ckpt(W, p, nck, st, tau);
                nck++;
            }
        }
    }
    cnt[C_TRAV]++; cnt[C_NBR] += st.nscanned(); cnt[C_FB] += st.fallbacks;
    if (st.steps > g.max_steps) { atomicOr(W.R.err, ERR_STEP_BUDGET); cnt[C_ERR]++; }
    double L = K.L, tau_int = 0;
    const int rc = after_path(W, S, p, phase, ell, tau, v2, L, tau_int);
    if (rc < 0) cnt[C_ERR]++;
    if (rc != 1) return;
    // DustGridPath::pathlength on the re-walked path
    double s = 0;
    bool resumed = false;
    if constexpr (CKPT) resumed = W.ckpt && resume_ckpt(W, g, p, nck, tau_int, st, tau, s);
    if (!resumed) {
        st.init(g, (R)K.x, (R)K.y, (R)K.z, (R)K.kx, (R)K.ky, (R)K.kz, K.pos_cell);
        R d0;
        while (st.pd.pop(d0)) s += (double)d0;
        tau = 0;
    }
    while (st.walk(g, m, ds)) {
        cnt[C_STEPS]++;
        const double tn = tau + step_dtau<R>(S, st, kext1, m, ell, ds), sn = s + (double)ds;
        if (tn > tau_int) {
            K.s_int = s + ((tau_int - tau) / (tn - tau)) * (sn - s);
            K.int_cell = m;
            K.state = PK_INTERACT;
            cnt[C_TRAV]++; cnt[C_NBR] += st.nscanned(); cnt[C_FB] += st.fallbacks;
            return;
        }
        tau = tn; s = sn;
    }
    cnt[C_TRAV]++; cnt[C_NBR] += st.nscanned(); cnt[C_FB] += st.fallbacks;
    if (st.steps > g.max_steps) { atomicOr(W.R.err, ERR_STEP_BUDGET); cnt[C_ERR]++; }
    K.s_int = s; K.int_cell = -1; K.state = PK_INTERACT;
}

// (4 blocks per SM, 128 registers: 10^4 packets on a 40x40x20 grid 0.90 ms against 1.40 at 2 blocks, 1.15 at 3;
// the Voronoi walk 9.9 ms at 3 against 12.9 at 4, 10^3 packets on 10^6 cells)
template<template<typename> class Stepper> struct TailBlocks { static constexpr int value = 4; };
template<> struct TailBlocks<VoronoiStepper> { static constexpr int value = 3; };
template<typename R, template<typename> class Stepper>
__global__ void __launch_bounds__(128, TailBlocks<Stepper>::value) tail_kernel(const WaveParams W) {
    const RunParams& P = W.R;
    // tail_lanes packets to a warp: few packets run side by side in few lanes, which then seldom
    // wait for one another's branches
    const int lane = threadIdx.x & 31;
    const int p = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * W.tail_lanes + lane;
    if (lane >= W.tail_lanes || p >= W.npool) return;
    Packet& K = W.pk[p];
    int state = K.state;
    if (state == PK_DONE) return;
    const BatchHeader H = *P.hdr;
    const int phase = H.phase;
    const bool peel_on = phase != SKG_PHASE_DUST_SELFABS;
    unsigned long long cnt[C_N];
    for (int c = 0; c < C_N; c++) cnt[c] = 0;
    while (true) {
        if (state == PK_INTERACT) {
            const WorkItem& It = P.items[K.item];
            const DevScene& S = *P.scenes[It.slot];
            const DevGrid& g = P.grids[It.slot];
            const R si = (R)K.s_int;                // PhotonPackage::propagate
            K.x = (double)((R)K.x + si * (R)K.kx);
            K.y = (double)((R)K.y + si * (R)K.ky);
            K.z = (double)((R)K.z + si * (R)K.kz);
            if (K.s_int > 0) K.pos_cell = (K.int_cell >= 0) ? K.int_cell : -2;
            const double kx0 = K.kx, ky0 = K.ky, kz0 = K.kz;
            if (peel_on) tail_peel<R, Stepper>(g, S, K, true, K.nscatt + 1, kx0, ky0, kz0, cnt, P.err);
            Philox rng;
            rng.init(It.seed, K.id, (uint32_t)K.ell | ((uint32_t)phase << 24));
            rng.c0 = K.rngc;
            const V3<double> kn = scatter_direction(S, K.ell, K.int_cell, mk3(K.kx, K.ky, K.kz), rng);
            K.rngc = rng.c0;
            K.kx = (double)(R)kn.x; K.ky = (double)(R)kn.y; K.kz = (double)(R)kn.z;
            K.nscatt++;
            cnt[C_SCATT]++;
            state = PK_WAIT;
        }
        if (state == PK_WAIT) {
            const int slot = P.items[K.item].slot;
            tail_path<R, Stepper>(W, P.grids[slot], *P.scenes[slot], p, phase, cnt);
            state = K.state;
            continue;
        }
        // a free record takes the next packet while there is one
        const unsigned long long gp = atomicAdd(P.work, 1ull);
        if (gp >= H.total) break;
        const int it = find_item(P.items, H.nitems, gp);
        const WorkItem It = P.items[it];
        const uint64_t q = gp - It.begin;
        const int ei = (int)(q / It.count);
        const uint64_t ip = It.first + (q - (uint64_t)ei * It.count);
        const int ell = P.ells[It.ell0 + ei];
        Philox rng;
        rng.init(It.seed, ip, (uint32_t)ell | ((uint32_t)phase << 24));
        cnt[C_PACKETS]++;
        const DevScene& S = *P.scenes[It.slot];
        const Launched o = launch_packet(P.grids[It.slot], S, phase, ell, It.npp_total, rng);
        state = PK_TERM;
        if (!o.ok) continue;
        K.x = (double)(R)o.x; K.y = (double)(R)o.y; K.z = (double)(R)o.z;
        K.kx = (double)(R)o.kx; K.ky = (double)(R)o.ky; K.kz = (double)(R)o.kz;
        K.L = o.L; K.Lth = o.Lth; K.s_int = 0;
        K.id = ip; K.item = it; K.ell = ell; K.nscatt = 0;
        K.pos_cell = -2; K.int_cell = -1; K.rngc = rng.c0;
        K.flags = pk_flags(o);
        if (peel_on) tail_peel<R, Stepper>(P.grids[It.slot], S, K, false, 0, 0, 0, 0, cnt, P.err);
        state = S.ncomp > 0 ? PK_WAIT : PK_TERM;   // without dust the life cycle ends here
    }
    K.state = PK_DONE;
    for (int c = 0; c < C_N; c++) if (cnt[c]) atomicAdd(P.counters + c, cnt[c]);
}

// ---------------------------------------------------------------------------------------------
// host side

namespace {

// SMs of the current device and the blocks of a kernel that are resident on it at once, for `smem`
// bytes of dynamic shared memory.  Above the 48 KB a kernel has by default (static and dynamic: the
// staged jobs and the grids of 58 and more slots on an FP64 walk) it is allowed them first.  Kept per
// device, kernel and size; a query that fails is reported and not kept.
struct Resident { int sms = 0, blocks = 0; };
cudaError_t resident(const void* kernel, int threads, size_t smem, Resident& out) {
    static std::mutex lock;
    static std::map<std::tuple<int, const void*, size_t>, Resident> known;
    int dev = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    std::lock_guard<std::mutex> hold(lock);
    const auto key = std::make_tuple(dev, kernel, smem);
    const auto it = known.find(key);
    if (it != known.end()) { out = it->second; return cudaSuccess; }
    cudaFuncAttributes attr;
    if ((e = cudaFuncGetAttributes(&attr, kernel)) != cudaSuccess) return e;
    if (smem > (size_t)std::max(attr.maxDynamicSharedSizeBytes, 0) &&
        (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    Resident r;
    int per = 0;
    if ((e = cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem)) != cudaSuccess) return e;
    if (per <= 0) return cudaErrorLaunchOutOfResources;
    r.blocks = r.sms * per;
    known[key] = r;
    out = r;
    return cudaSuccess;
}

// A traversal instantiation: persistent, so its blocks resident at once (or `blocks`, if given).  pdl: as a
// programmatic dependent of the kernel before it.
template<typename R, template<typename> class Stepper, int MODE, bool ONE>
cudaError_t launch_trav(const WaveParams& W, size_t smem, int blocks, bool pdl, cudaStream_t s) {
    Resident r;
    cudaError_t e = resident((const void*)trav_kernel<R, Stepper, MODE, ONE>, 256, smem, r);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks > 0 ? blocks : r.blocks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? SKG_PDL : 0;
    return cudaLaunchKernelEx(&cfg, trav_kernel<R, Stepper, MODE, ONE>, W);
}

// One wave: its kernels in order, none behind one that could not be launched (the ends of paths would
// tally optical depths that no walk wrote).
template<typename R, template<typename> class Stepper, bool ONE>
cudaError_t enqueue_wave(const WaveParams& W, int nslots, int trav_blocks, cudaEvent_t mid, cudaStream_t s) {
    const size_t smem = (size_t)nslots * sizeof(DevGrid);
    const int need = (W.npool + 255) / 256;
    // grid-stride passes over at most the blocks resident at once
    cudaError_t e;
    Resident l, d;
    if ((e = resident((const void*)launch_kernel<R>, 256, 0, l)) != cudaSuccess) return e;
    if ((e = resident((const void*)end_kernel, 256, 0, d)) != cudaSuccess) return e;
    launch_kernel<R><<<std::min(need, l.blocks), 256, 0, s>>>(W);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (W.hist) {
        bin_sums_kernel<<<2 * JOB_BINS / BIN_BLOCK, 1024, 0, s>>>(W.hist, W.bin0 + 2 * JOB_BINS);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        bins_kernel<<<2 * JOB_BINS / BIN_BLOCK, 1024, 0, s>>>(W.hist, W.bin0, W.bin0 + 2 * JOB_BINS);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        order_kernel<<<std::min(l.sms * 8, need), 256, 0, s>>>(W);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (mid && (e = cudaEventRecord(mid, s)) != cudaSuccess) return e;
    if (W.path_tau) {
        if ((e = launch_trav<R, Stepper, TRAV_TAU, ONE>(W, smem, trav_blocks, false, s)) != cudaSuccess) return e;
    } else {
        if ((e = launch_trav<R, Stepper, TRAV_PATH, ONE>(W, smem, trav_blocks, false, s)) != cudaSuccess) return e;
        if ((e = launch_trav<R, Stepper, TRAV_TAU, ONE>(W, smem, 0, true, s)) != cudaSuccess) return e;
    }
    end_kernel<<<std::min(need, d.blocks), 256, 0, s>>>(W);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // On large trees the few cells of the re-walks come from the lattice records, one table for all
    // directions: a wave's re-walks touch most of the eight octant tables once, and their records come
    // from DRAM (2.9 GB per launch on the 3*10^6-leaf octree).  2*10^7 packets there 190 -> 186 ms a
    // pass; 32 MB of records the same either way, a small octree 2.9 -> 3.0 ms.
    if constexpr (std::is_same<Stepper<R>, TreeOctantStepper<float>>::value)
        if (W.rewalk_lattice) return launch_trav<float, TreeLatticeStepper, TRAV_REWALK, ONE>(W, smem, 0, false, s);
    return launch_trav<R, Stepper, TRAV_REWALK, ONE>(W, smem, 0, false, s);
}

template<typename R, template<typename> class Stepper>
cudaError_t enqueue_tail(WaveParams W, cudaStream_t s) {
    if (W.wave == 0) {                // the whole phase: spread the packets over the warps resident at once
        Resident r;
        cudaError_t e = resident((const void*)tail_kernel<R, Stepper>, 128, 0, r);
        if (e != cudaSuccess) return e;
        W.tail_lanes = std::min(32, std::max(1, (W.npool + r.blocks * 4 - 1) / (r.blocks * 4)));
    }
    const int warps = (W.npool + W.tail_lanes - 1) / W.tail_lanes;
    tail_kernel<R, Stepper><<<(warps + 3) / 4, 128, 0, s>>>(W);
    return cudaGetLastError();
}

using WaveFn = cudaError_t (*)(const WaveParams&, int, int, cudaEvent_t, cudaStream_t);
using TailFn = cudaError_t (*)(WaveParams, cudaStream_t);
struct PassFns { WaveFn wave; TailFn tail; };

template<typename R, template<typename> class Stepper, bool ONE = false>
PassFns fns() { return {enqueue_wave<R, Stepper, ONE>, enqueue_tail<R, Stepper>}; }

// the FP32 tree and Voronoi walks have a single-slot instantiation (the grid as a kernel parameter:
// traversal pass of a phase, Voronoi disk 255 against 260 ms, k-d tree disk 1778 against 1800 ms,
// octree disk 1443 against 1445 ms; the Cartesian walk, 64.5 against 64.1 ms, keeps its shared copy)
template<template<typename> class Stepper>
PassFns fns32(bool one) { return one ? fns<float, Stepper, true>() : fns<float, Stepper, false>(); }

PassFns pick(int grid_type, int tree_walk, int precision, bool one) {
    const bool f64 = precision == SKG_PREC_FP64;
    switch (grid_type) {
    case SKG_GRID_CARTESIAN:
        if (f64) return fns<double, CartStepper>();
        return tree_walk == CW_UNIFORM ? fns<float, CartUniStepper>() : fns<float, CartStepper>();
    case SKG_GRID_OCTREE:
    case SKG_GRID_BINTREE:
        if (f64) return fns<double, TreeStepper>();
        if (tree_walk == TW_NODES) return fns<float, TreeNodeWalk>();
        if (tree_walk == TW_OCTANT) return fns32<TreeOctantStepper>(one);
        if (tree_walk == TW_LATTICE) return fns32<TreeLatticeStepper>(one);
        return fns32<TreeStepper>(one);
    default:
        return f64 ? fns<double, VoronoiStepper>() : fns32<VoronoiStepper>(one);
    }
}

}  // namespace

WaveRunner::~WaveRunner() {
    for (cudaEvent_t e : ev_) cudaEventDestroy(e);
    for (cudaEvent_t e : tail_ev_) if (e) cudaEventDestroy(e);
    // (a runner that never reserved frees nothing: no device-wide synchronisation)
    for (void* p : {(void*)pk_, (void*)lists_[0], (void*)lists_[1], (void*)rlist_, (void*)ckpt_, (void*)ctr_, (void*)bins_,
                    (void*)order_, (void*)jobs_, (void*)jtau_, (void*)jL_})
        if (p) cudaFree(p);
    if (h_ctr_) cudaFreeHost(h_ctr_);
    if (copied_) cudaEventDestroy(copied_);
}

// grids whose FP32 walk resumes from checkpoints (the steppers' Resumable trait)
static bool ckpt_grid(int grid_type) {
    if (grid_type == SKG_GRID_VORONOI) return Resumable<VoronoiStepper<float>>::value;
    if (grid_type == SKG_GRID_CARTESIAN) return Resumable<CartStepper<float>>::value;
    return Resumable<TreeLatticeStepper<float>>::value;
}

// Jobs in spatial order: the lanes of a warp walk through the same region, so more of the grid's
// records come from L1 and L2, for the cost of the counting sort.  Worth it when the wave has enough
// jobs to be dense and the records are more than what stays close anyway: phases of 2*10^7 packets on
// a 3*10^6-leaf octree (96 MB of records) 306 against 293 ms, of 2*10^6 on 10^6 Voronoi cells (512 MB)
// 262 against 254 ms, of 10^6 on the octree 20.7 against 18.3, on
// Voronoi cells 100 against 93, on a 10^6-leaf k-d tree 12.9 against 12.6; below these bounds the sort costs more than it gives
// (2.4*10^5 packets on a small octree 4.1 against 4.7 ms, 6*10^5 on the k-d tree 9.4 against 9.6; Cartesian
// densities are a few MB: a batch of 24 fit variants 53.5 against 56.2 ms).
static bool order_pays(int grid_type, size_t pool, size_t walk_bytes) {
    return grid_type != SKG_GRID_CARTESIAN && pool >= ((size_t)3 << 18) && pool < ((size_t)1 << 28) && walk_bytes >= ((size_t)8 << 20);
}

cudaError_t WaveRunner::reserve(size_t pool, int ngroups, int grid_type, size_t walk_bytes) {
    cudaError_t e;
    const size_t had[5] = {cap_pool_, cap_ckpt_, cap_jobs_, cap_order_, bins_ != nullptr};
    big_records_ = walk_bytes >= ((size_t)64 << 20);
    order_on_ = order_pays(grid_type, pool, walk_bytes);
    if (!ctr_) {
        if ((e = cudaMalloc(&ctr_, NCTR * sizeof(unsigned))) != cudaSuccess) return e;
        if ((e = cudaMallocHost((void**)&h_ctr_, NCTR * sizeof(unsigned))) != cudaSuccess) return e;
        if ((e = cudaEventCreateWithFlags(&copied_, cudaEventDisableTiming)) != cudaSuccess) return e;
    }
    if (pool > cap_pool_) {
        for (void** q : {(void**)&pk_, (void**)&lists_[0], (void**)&lists_[1], (void**)&rlist_}) { cudaFree(*q); *q = nullptr; }
        cap_pool_ = 0;
        if ((e = cudaMalloc(&pk_, pool * sizeof(Packet))) != cudaSuccess) return e;
        for (int b = 0; b < 2; b++)
            if ((e = cudaMalloc(&lists_[b], 2 * pool * sizeof(int))) != cudaSuccess) return e;
        if ((e = cudaMalloc(&rlist_, pool * sizeof(int2))) != cudaSuccess) return e;
        cap_pool_ = pool;
    }
    if (SKG_CKPT && ckpt_grid(grid_type) && pool > cap_ckpt_) {
        cudaFree(ckpt_); ckpt_ = nullptr; cap_ckpt_ = 0;
        if ((e = cudaMalloc(&ckpt_, pool * SKG_CKPT_N * 2 * sizeof(float4))) != cudaSuccess) return e;
        cap_ckpt_ = pool;
    }
    if (order_on_ && !bins_) {
        if ((e = cudaMalloc(&bins_, (4 * (size_t)JOB_BINS + 1024) * sizeof(unsigned))) != cudaSuccess) return e;
    }
    const size_t jobs = pool * (size_t)(ngroups + 1);
    if (jobs > cap_jobs_) {

        for (void** q : {(void**)&jobs_, (void**)&jtau_, (void**)&jL_}) { cudaFree(*q); *q = nullptr; }
        cap_jobs_ = 0;
        if ((e = cudaMalloc(&jobs_, jobs * sizeof(int2))) != cudaSuccess) return e;
        if ((e = cudaMalloc(&jtau_, jobs * sizeof(double))) != cudaSuccess) return e;
        if ((e = cudaMalloc(&jL_, jobs * sizeof(double))) != cudaSuccess) return e;
        cap_jobs_ = jobs;
    }
    if (order_on_ && jobs > cap_order_) {
        // (peel-off jobs, then the path jobs)
        cudaFree(order_); order_ = nullptr; cap_order_ = 0;
        if ((e = cudaMalloc(&order_, jobs * sizeof(uint2))) != cudaSuccess) return e;
        cap_order_ = jobs;
    }
    const size_t has[5] = {cap_pool_, cap_ckpt_, cap_jobs_, cap_order_, bins_ != nullptr};
    if (std::memcmp(had, has, sizeof(had)) != 0) generation_++;
    return cudaSuccess;
}

cudaError_t WaveRunner::enqueue(int n) {
    WaveFn fn = pick(ph_.grid_type, ph_.tree_walk, ph_.precision, ph_.one).wave;
    cudaError_t e;
    for (int i = 0; i < n; i++) {
        const int w = waves_ + i, b = w & 1;
        WaveParams W;
        W.R = ph_.P; W.pk = pk_; W.npool = ph_.npool; W.wave = w;
        W.jobs = jobs_; W.jtau = jtau_; W.jL = jL_;
        W.jcount = ctr_ + J_N * b; W.jnext = ctr_ + J_N * (b ^ 1);
        W.last_busy = ctr_ + 2 * J_N;
        W.freelist = lists_[b]; W.intlist = lists_[b] + ph_.npool; W.freenext = lists_[b ^ 1]; W.intnext = lists_[b ^ 1] + ph_.npool;
        W.rlist = rlist_; W.path_tau = ph_.path_tau; W.ckpt = ph_.ckpt_on ? ckpt_ : nullptr;
        W.g0 = ph_.g0;
        W.rewalk_lattice = ph_.tree_walk == TW_OCTANT && ph_.grid_type != SKG_GRID_CARTESIAN &&
                           ph_.precision == SKG_PREC_FP32 && ph_.big_records;
        W.hist = ph_.order_on ? bins_ : nullptr; W.bin0 = bins_ + 2 * JOB_BINS;
        // (a job's key lies where its optical depth will)
        W.jkey = reinterpret_cast<uint2*>(jtau_); W.speel = order_;
        W.spath = reinterpret_cast<int*>(order_ + (cap_order_ - ph_.npool));
        if ((e = cudaMemsetAsync(ctr_ + J_N * (b ^ 1), 0, J_N * sizeof(unsigned), stream_)) != cudaSuccess) return e;
        if (timed_) {
            while (ev_.size() < 3 * (size_t)(w + 1)) {
                cudaEvent_t x;
                if ((e = cudaEventCreate(&x)) != cudaSuccess) return e;
                ev_.push_back(x);
            }
            if ((e = cudaEventRecord(ev_[3 * w], stream_)) != cudaSuccess) return e;
        }
        if ((e = fn(W, ph_.nslots, ph_.trav_blocks, timed_ ? ev_[3 * w + 1] : nullptr, stream_)) != cudaSuccess) return e;
        if (timed_ && (e = cudaEventRecord(ev_[3 * w + 2], stream_)) != cudaSuccess) return e;
    }
    waves_ += n;
    if ((e = cudaMemcpyAsync(h_ctr_, ctr_, NCTR * sizeof(unsigned), cudaMemcpyDeviceToHost, stream_)) != cudaSuccess) return e;
    return record_copied();
}

cudaError_t WaveRunner::record_copied() {
    cudaError_t e;
    // inside stream capture the record must become a graph node that the host can wait on
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if ((e = cudaStreamIsCapturing(stream_, &cs)) != cudaSuccess) return e;
    return cs == cudaStreamCaptureStatusNone ? cudaEventRecord(copied_, stream_)
                                             : cudaEventRecordWithFlags(copied_, stream_, cudaEventRecordExternal);
}

cudaError_t WaveRunner::begin(const RunParams& P, int grid_type, int tree_walk, int precision, int nslots,
                              size_t npool, bool fits, int trav_blocks, bool absorbs, cudaStream_t s,
                              const DevGrid* one_grid) {
    const cudaError_t e = start(P, grid_type, tree_walk, precision, nslots, npool, fits, trav_blocks, absorbs, s, one_grid);
    return e == cudaSuccess ? e : over(e);
}

// A phase that could not be enqueued is over: nothing is added to it, what it had enqueued no longer uses
// the pool and its simulations' tables when the call returns, and its error is not a later call's.
cudaError_t WaveRunner::over(cudaError_t e) {
    pending_ = timed_ = false;
    cudaGetLastError();
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream_, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) cudaStreamSynchronize(stream_);
    cudaGetLastError();
    return e;
}

cudaError_t WaveRunner::start(const RunParams& P, int grid_type, int tree_walk, int precision, int nslots,
                              size_t npool, bool fits, int trav_blocks, bool absorbs, cudaStream_t s,
                              const DevGrid* one_grid) {
    stream_ = s;
    if (npool == 0 || npool > cap_pool_) return cudaErrorInvalidValue;
    ph_.P = P; ph_.grid_type = grid_type; ph_.tree_walk = tree_walk; ph_.precision = precision; ph_.nslots = nslots;
    ph_.one = one_grid != nullptr && nslots == 1;
    if (ph_.one) ph_.g0 = *one_grid; else std::memset(&ph_.g0, 0, sizeof(ph_.g0));
    ph_.trav_blocks = trav_blocks; ph_.npool = (int)npool; waves_ = 0; tail_ran_ = false;
    const char* td = std::getenv("SKG_TAIL_DIV");
    ph_.tail_div = td ? std::atoi(td) : tail_div;
    ph_.path_tau = !absorbs;
    ph_.order_on = order_on_; ph_.big_records = big_records_;
    const char* ck = std::getenv("SKG_CKPT");
    ph_.ckpt_on = !(ck && std::atoi(ck) == 0) && ckpt_ && cap_ckpt_ >= (size_t)npool;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cs);
    timed_ = timing && cs == cudaStreamCaptureStatusNone;
    cudaError_t e;
    if ((e = cudaMemsetAsync(ctr_, 0, NCTR * sizeof(unsigned), s)) != cudaSuccess) return e;
    // (the waves leave the counts of the bins at zero; cleared here, on the phase's stream, for the first and for
    // one that follows a failed phase)
    if (order_on_ && (e = cudaMemsetAsync(bins_, 0, 2 * JOB_BINS * sizeof(unsigned), s)) != cudaSuccess) return e;
    tail_only_ = ph_.tail_div > 0 && fits && npool <= (size_t)(grid_type == SKG_GRID_CARTESIAN ? SKG_TAIL_ONLY_CART : SKG_TAIL_ONLY);
    if (!tail_only_) {
        // (a divisor of 1 hands the phase over whatever the first look finds: it looks after one wave)
        if ((e = enqueue(ph_.tail_div == 1 ? 1 : estimate)) != cudaSuccess) return e;
    } else {
        if ((e = cudaMemsetAsync(pk_, 0, npool * sizeof(Packet), s)) != cudaSuccess) return e;   // (wave 0 writes every record)
        if ((e = enqueue_tail()) != cudaSuccess) return e;
        if ((e = record_copied()) != cudaSuccess) return e;
    }
    pending_ = cs == cudaStreamCaptureStatusNone;   // (a captured phase runs when it is replayed)
    return cudaSuccess;
}

cudaError_t WaveRunner::enqueue_tail() {
    WaveParams W;
    W.R = ph_.P; W.pk = pk_; W.npool = ph_.npool; W.wave = waves_;
    W.jobs = nullptr; W.jtau = nullptr; W.jL = nullptr; W.jcount = nullptr; W.jnext = nullptr;
    W.last_busy = ctr_ + 2 * J_N;
    W.tail_lanes = 32;
    W.freelist = nullptr; W.intlist = nullptr; W.freenext = nullptr; W.intnext = nullptr; W.rlist = nullptr; W.path_tau = 0; W.ckpt = ph_.ckpt_on ? ckpt_ : nullptr;
    W.rewalk_lattice = 0;
    W.hist = nullptr; W.bin0 = nullptr; W.jkey = nullptr; W.spath = nullptr; W.speel = nullptr;
    cudaError_t e;
    if (timed_) {
        for (int i = 0; i < 2; i++)
            if (!tail_ev_[i] && (e = cudaEventCreate(&tail_ev_[i])) != cudaSuccess) return e;
        if ((e = cudaEventRecord(tail_ev_[0], stream_)) != cudaSuccess) return e;
    }
    W.g0 = ph_.g0;
    if ((e = pick(ph_.grid_type, ph_.tree_walk, ph_.precision, ph_.one).tail(W, stream_)) != cudaSuccess) return e;
    tail_ran_ = true;
    return timed_ ? cudaEventRecord(tail_ev_[1], stream_) : cudaSuccess;
}

cudaError_t WaveRunner::finish(int timeout_ms, cudaEvent_t end, bool* timed_out) {
    if (timed_out) *timed_out = false;
    const auto t0 = std::chrono::steady_clock::now();
    bool more = false;                            // waves were added after the caller's end event
    while (pending_) {
        while (true) {
            const cudaError_t q = cudaEventQuery(copied_);
            if (q == cudaSuccess) break;
            if (q != cudaErrorNotReady) return q;
            if (timeout_ms >= 0 &&
                std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count() > timeout_ms) {
                if (timed_out) *timed_out = true;
                return cudaSuccess;
            }
            wait_a_little(t0, 50);
        }
        if (tail_only_) { pending_ = false; break; }
        // packets with jobs in the last wave (without dust a packet has peel-offs alone, or, off every
        // frame, no job at all: its record then waits on the next wave's free list)
        const unsigned* c = h_ctr_ + J_N * ((waves_ - 1) & 1);
        const unsigned busy = c[J_PATH] ? c[J_PATH] : c[J_PEEL];
        if (busy == 0 && h_ctr_[J_N * (waves_ & 1) + J_FREE] == 0) {
            pending_ = false;
            estimate = (int)h_ctr_[2 * J_N] + 2;        // the last busy wave, the empty one, one spare
            break;
        }
        if (ph_.tail_div > 0 && (size_t)busy * (size_t)ph_.tail_div <= (size_t)ph_.npool) {
            // few packets left in flight: the tail pass finishes them (and any packets still to
            // launch) in one launch; the next phase enqueues this many waves before it looks
            cudaError_t e = enqueue_tail();
            if (e != cudaSuccess) return over(e);
            pending_ = false;
            if (ph_.tail_div != 1) estimate = waves_;
            more = true;
            break;
        }
        cudaError_t e = enqueue(estimate > 32 ? estimate / 4 : 8);
        if (e != cudaSuccess) return over(e);
        more = true;
    }
    return (end && more) ? cudaEventRecord(end, stream_) : cudaSuccess;
}

cudaError_t WaveRunner::times(float* event_ms, float* trav_ms) const {
    float a = 0, t = 0;
    if (timed_ && !pending_) {
        for (int w = 0; w < waves_; w++) {
            float x = 0, y = 0;
            cudaError_t e = cudaEventElapsedTime(&x, ev_[3 * w], ev_[3 * w + 1]);
            if (e == cudaSuccess) e = cudaEventElapsedTime(&y, ev_[3 * w + 1], ev_[3 * w + 2]);
            if (e != cudaSuccess) return e;
            a += x; t += y;
        }
        if (tail_ran_) {
            float y = 0;
            cudaError_t e = cudaEventElapsedTime(&y, tail_ev_[0], tail_ev_[1]);
            if (e != cudaSuccess) return e;
            t += y;
        }
    }
    if (event_ms) *event_ms = a;
    if (trav_ms) *trav_ms = t;
    return cudaSuccess;
}

}  // namespace skg
