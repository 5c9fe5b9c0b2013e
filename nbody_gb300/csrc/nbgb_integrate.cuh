// nbgb_integrate.cuh -- the reference integrator as a force kernel's epilogue.
#pragma once

#include "nbgb_device.cuh"
#include "nbgb_internal.h"

namespace nbgb {

// The reference integrator (integrateOne, src/nbody.cu:158-182) applied to
// target i by the unit that produced its final force F: v += (F invMass) dt;
// v *= damping; x += v dt, each operation rounded separately or, fused drift,
// x = fma(v, dt, x) -- the same arithmetic as integrate_reference_kernel, so
// the results are identical.  Writes posMass (mass kept), velInvMass and body
// i's entry of the next step's j-stream (fi.js, the other buffer: the current
// one is still being read by other units; fi.js == nullptr: no j-stream is
// kept, the pair kernel reads posMass).  Only the last unit of an
// i-block writes its targets, after every unit of that i-block has loaded
// them, so no unit reads a target this launch has moved.
// v: the body's velInvMass.
__device__ __forceinline__ void fused_integrate(const FusedIntegrate &fi, int i, float4 v, float x,
                                                float y, float z, float m, float fx, float fy,
                                                float fz) {
    const float im = v.w, dt = fi.dt;
    v.x = __fmul_rn(__fadd_rn(v.x, __fmul_rn(__fmul_rn(fx, im), dt)), fi.damping);
    v.y = __fmul_rn(__fadd_rn(v.y, __fmul_rn(__fmul_rn(fy, im), dt)), fi.damping);
    v.z = __fmul_rn(__fadd_rn(v.z, __fmul_rn(__fmul_rn(fz, im), dt)), fi.damping);
    if (fi.fused_drift) {
        x = __fmaf_rn(v.x, dt, x);
        y = __fmaf_rn(v.y, dt, y);
        z = __fmaf_rn(v.z, dt, z);
    } else {
        x = __fadd_rn(x, __fmul_rn(v.x, dt));
        y = __fadd_rn(y, __fmul_rn(v.y, dt));
        z = __fadd_rn(z, __fmul_rn(v.z, dt));
    }
    fi.pm[i] = make_float4(x, y, z, m);
    fi.vel[i] = v;
    if (!fi.js)
        return;
    const int q = i >> 1, h = i & 1;
    float w = m;
    if (fi.js_log && jstream_log_slot(q))
        w = jstream_log_mass(w);
    if (fi.js_vpb == 2) {
        fi.js[2 * i] = make_float4(x, x, y, y);
        fi.js[2 * i + 1] = make_float4(z, z, w, w);
    } else {
        float *a = reinterpret_cast<float *>(fi.js + 2 * q);
        a[h] = x;
        a[2 + h] = y;
        a[4 + h] = z;
        a[6 + h] = w;
    }
}

}  // namespace nbgb
