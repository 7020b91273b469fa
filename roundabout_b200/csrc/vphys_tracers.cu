// vphys_tracers.cu -- the exact tracer solve (vphys_tracers.cuh) in groups of up to
// five tracers a thread, its launcher, and the FP64 re-solve for the mixed form.
#include <cuda_runtime.h>

#include "vphys_tracers.cuh"

namespace vphys {

// Groups of at most VPHYS_TR_GROUP tracers, as even as they come: a thread's
// registers hold one group, and each group repeats the factorisation.  Over a few
// levels a thread's time is its set-up (the span scans, the column scalars, the
// round trips of the first loads), which each group repeats too: there one thread
// takes every tracer, a level a block, where the grid has the columns to fill the
// chip.  us on 300x300 columns with groups / one thread:
//   default knobs, one factorisation and two
//     1 level    6 tracers 18.8 / 14.6 and 23.1 / 14.8    16: 40.9 / 26.0 and 54.2 / 27.2
//     8 levels   6: 36.9 / 33.2 and 47.8 / 39.1           16: 86.5 / 63.0 and 122.5 / 76.2
//     50 levels  6: 155.9 / 173.4                         16: 340.7 / 393.4
//   two full groups of five: 10 tracers 37.3 / 37.9 at 4 levels, 50.0 / 53.9 at 8
//   budgets      8 tracers 72.9 / 61.0 at 8 levels        16: 68.6 / 62.4 at 3, 108.1 / 111.3 at 6
//   content      8 tracers 91.7 / 75.4 at 8 levels        16: 99.2 / 109.1 at 3 (registers)
// 64x64 columns leave most of the chip to the groups (20 levels, 16 tracers 18.8 / 33.2).
inline int tracer_groups(const Params &p, bool fills, bool diffuse)
{
    int shallow = 8;
    if (p.ntr > 8) {
        if (is_default_tracer_knobs(p.cfg))
            shallow = p.ntr > 10 ? 8 : 4;
        else
            shallow = (p.ntr > 10 && !(p.content_old && diffuse)) ? 3 : 0;
    }
    if (fills && p.nz <= shallow) return 1;
    return (p.ntr + VPHYS_TR_GROUP - 1) / VPHYS_TR_GROUP;
}

// The FP64 re-solve of the (32-column group, tracer) pairs that the
// mixed-precision kernel listed (mp_redo[0] entries after the count, each
// group << 5 | tracer) and left untouched: each runs the exact path above as
// a one-tracer problem -- the tracer's roles (T, S, pseudo-salt) and its
// diffusivity carried over -- so those columns come out bitwise as on the
// FP64 path.  One warp per entry, the grid strides over the list.
__global__ void __launch_bounds__(32) k_tracers_redo(const Params p, double dt, int nonlocal, int ngx)
{
    extern __shared__ double smem[];
    const unsigned n = *(volatile const unsigned *)p.mp_redo;
    for (unsigned e = blockIdx.x; e < n; e += gridDim.x) {
        const unsigned ent = p.mp_redo[1 + e];
        const int tix = (int)(ent & 31u);
        const unsigned g = ent >> 5;
        const int gi = (int)(g % (unsigned)ngx), j = (int)(g / (unsigned)ngx);
        const int li = gi * 32 + (int)threadIdx.x;
        Params q = p;
        const vphys_config &c = p.cfg;
        q.ntr = 1;
        q.tr[0] = p.tr[tix];
        q.cfg.idx_temperature = (tix == c.idx_temperature) ? 0 : -1;
        q.cfg.idx_salinity = (tix == c.idx_salinity) ? 0 : -1;
        q.cfg.idx_pseudo_salt = (tix == c.idx_pseudo_salt) ? 0 : -1;
        if (!p.ks_equals_kt && tix != c.idx_temperature) q.kt = p.ks;   // the second factorisation's tracers
        if (p.content_old) {
            q.content_old = p.content_old + p.plane * (size_t)tix;   // the tracer's plane of the content fields
            q.content_new = p.content_new + p.plane * (size_t)tix;
            tracer_columns<1, false, false, true>(q, dt, 1, nonlocal, li, j, smem, threadIdx.x, 32);
        } else {
            tracer_columns<1, false, false>(q, dt, 1, nonlocal, li, j, smem, threadIdx.x, 32);
        }
        __syncwarp();
    }
}

static void redo_attr()
{
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_tracers_redo, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((size_t)VPHYS_NZ_MAX * 32 * sizeof(double)));
        attr_set = true;
    }
}

void launch_tracers_redo(const Params &p, double dt, bool nonlocal, cudaStream_t stream)
{
    redo_attr();
    const int ngx = (p.nx + 31) / 32;
    const size_t smem = (size_t)p.nz * 32 * sizeof(double);
    k_tracers_redo<<<148 * 8, 32, smem, stream>>>(p, dt, nonlocal ? 1 : 0, ngx);
}

template <bool TWO>
static void launch_tracers_g(const Params &p, double dt, bool diffuse, bool nonlocal, cudaStream_t stream)
{
    const bool fills = (long long)((p.nx + VPHYS_TR_THREADS - 1) / VPHYS_TR_THREADS) * p.ny > 148;
    const int ngroups = tracer_groups(p, fills, diffuse);
    switch ((p.ntr + ngroups - 1) / ngroups) {
    case 1: launch_tracers_n<1, TWO>(p, dt, diffuse, nonlocal, ngroups, stream); break;
    case 2: launch_tracers_n<2, TWO>(p, dt, diffuse, nonlocal, ngroups, stream); break;
    case 3: launch_tracers_n<3, TWO>(p, dt, diffuse, nonlocal, ngroups, stream); break;
    case 4: launch_tracers_n<4, TWO>(p, dt, diffuse, nonlocal, ngroups, stream); break;
    case 5: launch_tracers_n<5, TWO>(p, dt, diffuse, nonlocal, ngroups, stream); break;
    default: launch_tracers_wide(p, dt, diffuse, nonlocal, TWO, stream); break;
    }
}

void launch_tracers(const Params &p, double dt, bool diffuse, bool nonlocal, cudaStream_t stream)
{
    if (p.ntr < 1) return;
    if (diffuse && p.cfg.mixed_precision) {
        launch_tracers_mp(p, dt, nonlocal, stream);
        return;
    }
    if (p.ks_equals_kt)
        launch_tracers_g<false>(p, dt, diffuse, nonlocal, stream);
    else
        launch_tracers_g<true>(p, dt, diffuse, nonlocal, stream);
}

}  // namespace vphys
