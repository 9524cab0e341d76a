// gy_export.cu -- particle fields from the slab's order and types to the getters': FP64 (or int),
// one row per particle in insertion order.
//
// A getter used to copy the whole slab (33 fields) to the host and convert the wanted one there,
// particle by particle in slot order: 39 ms for the positions and 25 ms for the velocities of 2.4
// million particles.  The kernel converts and orders on the device, and only the rows the caller
// asked for cross to the host.  It is bound by that copy.
#include <algorithm>

#include "../../include/graphyt_gpu.h"
#include "gy_kernels.cuh"

namespace gy {

// FP64 operations rounded one by one, as the conversion is defined
__device__ __forceinline__ double moved(int c, int c0, float o, float o0, double h)
{
    return __dmul_rn((double)(c - c0) + ((double)o - (double)o0), h);
}

__device__ __forceinline__ int ref_cell(int ix, int iy, int iz, const GridGeom &g)
{
    return ix + iy * (g.nx - 1) + iz * (g.nx - 1) * (g.ny - 1);
}

__global__ void __launch_bounds__(256) k_export(PView P, long long n, int field, ExportArgs a, double *out)
{
    const GridGeom &g = a.g;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long pid = P.ii(PF_PID, i);
        auto rows = [&](int f, int w, bool on) {
            for (int k = 0; k < w; k++) out[pid * w + k] = on ? (double)P.f(f + k, i) : 0.0;
        };
        switch (field) {
        case GY_P_POS:
        case GY_P_DISP: {
            // displacement from the change of (cell, FP32 offset) since upload, so that a particle
            // that has not moved reports exactly zero; position = pos0 + disp
            int c[3], c0[3];
            decode_key(P.ii(PF_KEY, i), g, c[0], c[1], c[2]);
            decode_key(a.key0[pid], g, c0[0], c0[1], c0[2]);
            for (int k = 0; k < 3; k++) {
                const double d =
                    k < 2 || g.is3d ? moved(c[k], c0[k], P.f(PF_OX + k, i), a.off0[k * P.cap + pid], a.h) : 0.0;
                out[3 * pid + k] = field == GY_P_POS ? __dadd_rn(a.pos0[3 * pid + k], d) : d;
            }
            break;
        }
        case GY_P_POS0: for (int k = 0; k < 3; k++) out[3 * pid + k] = a.pos0[3 * pid + k]; break;
        case GY_P_VEL: rows(PF_VX, 3, true); break;
        case GY_P_STRESS: rows(PF_S0, 6, true); break;
        case GY_P_STRAIN: rows(PF_E0, 6, true); break;
        case GY_P_PSTRAIN: rows(PF_EP0, 6, a.has_dp); break;
        case GY_P_EQPS: rows(PF_EQPS, 1, a.has_dp); break;
        case GY_P_DAMAGE: rows(PF_DMG, 1, a.has_dp); break;
        case GY_P_SMAX: rows(PF_SMAX, 1, a.has_dp); break;
        case GY_P_MASS: rows(PF_MASS, 1, true); break;
        case GY_P_DENSITY: rows(PF_RHO, 1, true); break;
        case GY_P_VOLUME:
            out[pid] = ((uint32_t)P.ii(PF_INFO, i) & INFO_INIT_VOL)
                           ? a.init_volume
                           : __ddiv_rn((double)P.f(PF_MASS, i), (double)P.f(PF_RHO, i));
            break;
        case GY_P_NORMALS: rows(PF_NX, 3, a.normals); break;
        default: break;
        }
    }
}

__global__ void __launch_bounds__(256) k_export_int(PView P, long long n, int field, ExportArgs a, int *out)
{
    const GridGeom &g = a.g;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long pid = P.ii(PF_PID, i);
        const uint32_t info = (uint32_t)P.ii(PF_INFO, i);
        switch (field) {
        case GY_PI_MATERIAL: out[pid] = info_mat(info); break;
        case GY_PI_OBJECT: out[pid] = a.slot_obj[info_obj(info)]; break;
        case GY_PI_DEVICE_SLOT: out[pid] = (int)i; break;
        case GY_PI_CELLID: {
            int id[3] = {0, 0, 0};
            if (info & INFO_INIT_VOL) {
                // no update yet: the initial unshifted key (MaterialPoints.cpp:228-231)
                for (int k = 0; k < 3; k++) id[k] = (int)__ddiv_rn(a.pos0[3 * pid + k], a.h);
            } else {
                int c[3];
                decode_key(P.ii(PF_KEY, i), g, c[0], c[1], c[2]);
                for (int k = 0; k < (g.is3d ? 3 : 2); k++) id[k] = (int)((c[k] + (double)P.f(PF_OX + k, i)) - 0.25);
            }
            out[pid] = ref_cell(id[0], id[1], id[2], g);
            break;
        }
        default: break;
        }
    }
}

// temperature (field GY_P_TEMP) or its gradient, kept by insertion index
__global__ void __launch_bounds__(256) k_export_therm(const float4 *therm, long long n, int field, double *out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 t = therm[i];
        if (field == GY_P_TEMP) {
            out[i] = t.x;
        } else {
            out[3 * i] = t.y;
            out[3 * i + 1] = t.z;
            out[3 * i + 2] = t.w;
        }
    }
}

static unsigned export_grid(long long n) { return (unsigned)std::max(1ll, std::min((n + 255) / 256, 65536ll)); }

cudaError_t launch_export(const PView &p, long long n, int field, const ExportArgs &a, double *out, cudaStream_t s)
{
    note_launch(1);
    return launch_checked(k_export, export_grid(n), 256, s, p, n, field, a, out);
}

cudaError_t launch_export_int(const PView &p, long long n, int field, const ExportArgs &a, int *out, cudaStream_t s)
{
    note_launch(1);
    return launch_checked(k_export_int, export_grid(n), 256, s, p, n, field, a, out);
}

cudaError_t launch_export_therm(const float4 *therm, long long n, int field, double *out, cudaStream_t s)
{
    note_launch(1);
    return launch_checked(k_export_therm, export_grid(n), 256, s, therm, n, field, out);
}

}  // namespace gy
