// fire_config.cu -- kernels of the config physics (FirePhysicsParams.mode 1).
//
// A plain T/F/S smoke-and-fire model on the same MAC grid and projection as
// the reference physics: semi-Lagrangian advection in cell units, first-order
// burn, seeded disk emitters, vorticity confinement, curl of seeded value
// noise, wind, and a point-light transmittance render.  The reference has
// none of these (its model is the ten-scalar fuel bed of src/fire_cuda.cu);
// the equations are stated in include/fire_ext.h.  The divergence, the SOR
// solve and the gradient subtraction are the reference-physics kernels.
//
// This file is compiled with -fmad=false: every product and sum rounds as
// written, and the only fused multiply-adds are the explicit ones of the
// interpolations (lerp1), so a CPU restatement that evaluates the same
// expressions in the same order in IEEE float, with std::fma where the
// kernels fuse, gives the same bits for the whole simulation step (only +, -,
// *, /, fma, sqrt, floor, min/max and integer hashing occur there).
// The render uses expf and is compared within a tolerance.
//
// Memory: records are read and written through the storage accessors
// (ldv/stv), so the FP16 and BF16 storage builds apply unchanged.  Only record
// a = (heat, fuel, oxygen, soot) is advanced; b and c are not touched.
#include "fire_kernels.h"

namespace firesim {

namespace {

__device__ __forceinline__ int faceIndex(int x, int y, int z, int mx, int my) { return (z * my + y) * mx + x; }

// Clamped trilinear sample of a grid of mx*my*mz values (x fastest) at index-space
// position q: q clamped to [0, m-1] per axis, i0 = (int)q, i1 = min(i0 + 1, m - 1),
// t = q - i0; lerp(a, b, t) = fma(t, b - a, a), along x, then y, then z.
struct Corners {
    int x0, x1, y0, y1, z0, z1;
    float tx, ty, tz;
};

__device__ __forceinline__ void axisOf(float q, int m, int& i0, int& i1, float& t) {
    q = fminf(fmaxf(q, 0.0f), static_cast<float>(m - 1));
    i0 = static_cast<int>(q);
    i1 = min(i0 + 1, m - 1);
    t = q - static_cast<float>(i0);
}

__device__ __forceinline__ Corners cornersAt(float qx, float qy, float qz, int mx, int my, int mz) {
    Corners c;
    axisOf(qx, mx, c.x0, c.x1, c.tx);
    axisOf(qy, my, c.y0, c.y1, c.ty);
    axisOf(qz, mz, c.z0, c.z1, c.tz);
    return c;
}

// One fused multiply-add (explicit, as the file is built without contraction).
__device__ __forceinline__ float lerp1(float a, float b, float t) { return __fmaf_rn(t, b - a, a); }

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t) {
    return make_float4(lerp1(a.x, b.x, t), lerp1(a.y, b.y, t), lerp1(a.z, b.z, t), lerp1(a.w, b.w, t));
}

// The eight corner loads address one base cell plus fixed offsets (0 or 1
// cell along each axis, 0 where the clamp merges the corners), which saves
// the index arithmetic of a full (z * my + y) * mx + x per corner.
template <typename P>
__device__ __forceinline__ float trilinear1(const P* f, const Corners& c, int mx, int my) {
    const P* b = f + faceIndex(c.x0, c.y0, c.z0, mx, my);
    const int dx = c.x1 - c.x0, dy = (c.y1 - c.y0) * mx, dz = (c.z1 - c.z0) * mx * my;
    const float a00 = lerp1(ldv(b), ldv(b + dx), c.tx);
    const float a10 = lerp1(ldv(b + dy), ldv(b + dy + dx), c.tx);
    const float a01 = lerp1(ldv(b + dz), ldv(b + dz + dx), c.tx);
    const float a11 = lerp1(ldv(b + dz + dy), ldv(b + dz + dy + dx), c.tx);
    const float b0 = lerp1(a00, a10, c.ty);
    const float b1 = lerp1(a01, a11, c.ty);
    return lerp1(b0, b1, c.tz);
}

__device__ __forceinline__ float4 trilinearRec(const Rec4* f, const Corners& c, int mx, int my) {
    const Rec4* b = f + faceIndex(c.x0, c.y0, c.z0, mx, my);
    const int dx = c.x1 - c.x0, dy = (c.y1 - c.y0) * mx, dz = (c.z1 - c.z0) * mx * my;
    const float4 a00 = lerp4(ldv(b), ldv(b + dx), c.tx);
    const float4 a10 = lerp4(ldv(b + dy), ldv(b + dy + dx), c.tx);
    const float4 a01 = lerp4(ldv(b + dz), ldv(b + dz + dx), c.tx);
    const float4 a11 = lerp4(ldv(b + dz + dy), ldv(b + dz + dy + dx), c.tx);
    const float4 b0 = lerp4(a00, a10, c.ty);
    const float4 b1 = lerp4(a01, a11, c.ty);
    return lerp4(b0, b1, c.tz);
}

// Velocity (cells per step) at the faces and cell centres the advection
// traces back from.  u lives at (i, j+.5, k+.5), v at (i+.5, j, k+.5), w at
// (i+.5, j+.5, k); the velocity at a point is the clamped trilinear sample of
// each face grid (x, then y, then z).  At these points one or two of each
// sample's weights are 0, and lerp(a, b, 0) = a, so those axes are skipped and
// the remaining lerps are taken in the same order: for finite velocities the
// values equal the full trilinear samples, except possibly in the sign of a
// zero, which the callers (position - velocity, position >= 0) cannot see.
__device__ __forceinline__ float faceAt(const FaceT* f, int x, int y, int z, int mx, int my) { return ldv(f + faceIndex(x, y, z, mx, my)); }

// At the u face (x, y + .5, z + .5).
__device__ __forceinline__ float3 velocityAtUFace(const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    int x0, x1;
    float tx;
    axisOf(static_cast<float>(x) - 0.5f, p.nx, x0, x1, tx);
    // v at y and y + 1 (weight 1/2), w at z and z + 1 (weight 1/2), x0 and x1 along x.
    const int dx = x1 - x0;
    const FaceT* vb = vel.v + faceIndex(x0, y, z, p.nx, p.ny + 1);
    const FaceT* wb = vel.w + faceIndex(x0, y, z, p.nx, p.ny);
    const int vy = p.nx, wz = p.nx * p.ny;
    const float v = lerp1(lerp1(ldv(vb), ldv(vb + dx), tx), lerp1(ldv(vb + vy), ldv(vb + vy + dx), tx), 0.5f);
    const float w = lerp1(lerp1(ldv(wb), ldv(wb + dx), tx), lerp1(ldv(wb + wz), ldv(wb + wz + dx), tx), 0.5f);
    return make_float3(faceAt(vel.u, x, y, z, p.nx + 1, p.ny), v, w);
}

// At the v face (x + .5, y, z + .5).
__device__ __forceinline__ float3 velocityAtVFace(const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    int y0, y1;
    float ty;
    axisOf(static_cast<float>(y) - 0.5f, p.ny, y0, y1, ty);
    const FaceT* ub = vel.u + faceIndex(x, y0, z, p.nx + 1, p.ny);
    const FaceT* wb = vel.w + faceIndex(x, y0, z, p.nx, p.ny);
    const int du = (y1 - y0) * (p.nx + 1), dw = (y1 - y0) * p.nx, wz = p.nx * p.ny;
    const float u = lerp1(lerp1(ldv(ub), ldv(ub + 1), 0.5f), lerp1(ldv(ub + du), ldv(ub + du + 1), 0.5f), ty);
    const float w = lerp1(lerp1(ldv(wb), ldv(wb + dw), ty), lerp1(ldv(wb + wz), ldv(wb + wz + dw), ty), 0.5f);
    return make_float3(u, faceAt(vel.v, x, y, z, p.nx, p.ny + 1), w);
}

// At the w face (x + .5, y + .5, z).
__device__ __forceinline__ float3 velocityAtWFace(const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    int z0, z1;
    float tz;
    axisOf(static_cast<float>(z) - 0.5f, p.nz, z0, z1, tz);
    const FaceT* ub = vel.u + faceIndex(x, y, z0, p.nx + 1, p.ny);
    const FaceT* vb = vel.v + faceIndex(x, y, z0, p.nx, p.ny + 1);
    const int du = (z1 - z0) * (p.nx + 1) * p.ny, dv = (z1 - z0) * p.nx * (p.ny + 1), vy = p.nx;
    const float u = lerp1(lerp1(ldv(ub), ldv(ub + 1), 0.5f), lerp1(ldv(ub + du), ldv(ub + du + 1), 0.5f), tz);
    const float v = lerp1(lerp1(ldv(vb), ldv(vb + vy), 0.5f), lerp1(ldv(vb + dv), ldv(vb + dv + vy), 0.5f), tz);
    return make_float3(u, v, faceAt(vel.w, x, y, z, p.nx, p.ny));
}

// At the cell centre (x + .5, y + .5, z + .5): the mean of the two faces along each axis.
__device__ __forceinline__ float3 velocityAtCentre(const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    const FaceT* ub = vel.u + faceIndex(x, y, z, p.nx + 1, p.ny);
    const FaceT* vb = vel.v + faceIndex(x, y, z, p.nx, p.ny + 1);
    const FaceT* wb = vel.w + faceIndex(x, y, z, p.nx, p.ny);
    return make_float3(lerp1(ldv(ub), ldv(ub + 1), 0.5f), lerp1(ldv(vb), ldv(vb + p.nx), 0.5f), lerp1(ldv(wb), ldv(wb + p.nx * p.ny), 0.5f));
}

__device__ __forceinline__ Corners recordCorners(const ConfigParams& p, float x, float y, float z) {
    return cornersAt(x - 0.5f, y - 0.5f, z - 0.5f, p.nx, p.ny, p.nz);
}
__device__ __forceinline__ float4 recordAt(const Rec4* a, const ConfigParams& p, float x, float y, float z) {
    return trilinearRec(a, recordCorners(p, x, y, z), p.nx, p.ny);
}

// Whether the brick of a sample's first corner holds something.
__device__ __forceinline__ bool brickSeen(const CfgOccupancy* occ, const Corners& c, int bx, int by) {
    return reinterpret_cast<const unsigned char*>(occ + 1)[((c.z0 >> 2) * by + (c.y0 >> 2)) * bx + (c.x0 >> 2)] != 0;
}

__device__ __forceinline__ bool inDisk(const ConfigEmitter& e, int x, int y, int z) {
    if (y != e.row) return false;
    const float dx = static_cast<float>(x) - e.cx;
    const float dz = static_cast<float>(z) - e.cz;
    return dx * dx + dz * dz <= e.r2;
}

// psi_c at position (x, y, z) (cell units) and its gradient: value noise on a
// lattice of period 1/invPeriod cells, cubic Hermite weights s = f^2 (3 - 2f),
// ds/df = 6 f (1 - f).
__device__ __forceinline__ float3 noiseGradient(const ConfigParams& p, int comp, float x, float y, float z) {
    const float qx = x * p.invPeriod, qy = y * p.invPeriod, qz = z * p.invPeriod;
    const float fx0 = floorf(qx), fy0 = floorf(qy), fz0 = floorf(qz);
    const int ix = static_cast<int>(fx0), iy = static_cast<int>(fy0), iz = static_cast<int>(fz0);
    const float fx = qx - fx0, fy = qy - fy0, fz = qz - fz0;
    const float sx = fx * fx * (3.0f - 2.0f * fx), sy = fy * fy * (3.0f - 2.0f * fy), sz = fz * fz * (3.0f - 2.0f * fz);
    const float dsx = 6.0f * fx * (1.0f - fx), dsy = 6.0f * fy * (1.0f - fy), dsz = 6.0f * fz * (1.0f - fz);
    const float c000 = latticeValue(p.noiseSeed, comp, ix, iy, iz), c100 = latticeValue(p.noiseSeed, comp, ix + 1, iy, iz);
    const float c010 = latticeValue(p.noiseSeed, comp, ix, iy + 1, iz), c110 = latticeValue(p.noiseSeed, comp, ix + 1, iy + 1, iz);
    const float c001 = latticeValue(p.noiseSeed, comp, ix, iy, iz + 1), c101 = latticeValue(p.noiseSeed, comp, ix + 1, iy, iz + 1);
    const float c011 = latticeValue(p.noiseSeed, comp, ix, iy + 1, iz + 1), c111 = latticeValue(p.noiseSeed, comp, ix + 1, iy + 1, iz + 1);
    const float a00 = lerp1(c000, c100, sx), a10 = lerp1(c010, c110, sx), a01 = lerp1(c001, c101, sx), a11 = lerp1(c011, c111, sx);
    const float b0 = lerp1(a00, a10, sy), b1 = lerp1(a01, a11, sy);
    const float e0 = lerp1(c100 - c000, c110 - c010, sy), e1 = lerp1(c101 - c001, c111 - c011, sy);
    const float gx = dsx * lerp1(e0, e1, sz);
    const float gy = dsy * lerp1(a10 - a00, a11 - a01, sz);
    const float gz = dsz * (b1 - b0);
    return make_float3(gx * p.invPeriod, gy * p.invPeriod, gz * p.invPeriod);
}

__device__ __forceinline__ float cellCentred(const FaceT* f, int lo, int hi) { return 0.5f * (ldv(f + lo) + ldv(f + hi)); }

}  // namespace

// Each thread owns u(x,y,z), v(x,y,z) and w(x,y,z) where they exist and
// writes each as the face grid sampled at its one-step backtrace.
__device__ __forceinline__ void cfgAdvectVelocityAt(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                         const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    const float fx = static_cast<float>(x), fy = static_cast<float>(y), fz = static_cast<float>(z);
    if (y < p.ny && z < p.nz) {
        const float px = fx, py = fy + 0.5f, pz = fz + 0.5f;
        const float3 d = velocityAtUFace(vel, p, x, y, z);
        const float bx = px - d.x, by = py - d.y, bz = pz - d.z;
        stv(uOut + faceIndex(x, y, z, p.nx + 1, p.ny),
            trilinear1(vel.u, cornersAt(bx, by - 0.5f, bz - 0.5f, p.nx + 1, p.ny, p.nz), p.nx + 1, p.ny));
    }
    if (x < p.nx && z < p.nz) {
        const float px = fx + 0.5f, py = fy, pz = fz + 0.5f;
        const float3 d = velocityAtVFace(vel, p, x, y, z);
        const float bx = px - d.x, by = py - d.y, bz = pz - d.z;
        stv(vOut + faceIndex(x, y, z, p.nx, p.ny + 1), trilinear1(vel.v, cornersAt(bx - 0.5f, by, bz - 0.5f, p.nx, p.ny + 1, p.nz), p.nx, p.ny + 1));
    }
    if (x < p.nx && y < p.ny) {
        const float px = fx + 0.5f, py = fy + 0.5f, pz = fz;
        const float3 d = velocityAtWFace(vel, p, x, y, z);
        const float bx = px - d.x, by = py - d.y, bz = pz - d.z;
        stv(wOut + faceIndex(x, y, z, p.nx, p.ny), trilinear1(vel.w, cornersAt(bx - 0.5f, by - 0.5f, bz, p.nx, p.ny, p.nz + 1), p.nx, p.ny));
    }
}

// The single-scene face kernels run on the cell grid: the thread of cell
// (x, y, z) owns its u, v and w faces and, as the last cell of its row,
// column or plane, the far wall's face beside it (x = nx, y = ny, z = nz).
// A face grid of nx + 1 columns would leave a nearly empty block per row.
template <class Face>
__device__ __forceinline__ void facesOfCell(const ConfigParams& p, int x, int y, int z, Face face) {
    face(x, y, z);
    if (x == p.nx - 1) face(p.nx, y, z);
    if (y == p.ny - 1) face(x, p.ny, z);
    if (z == p.nz - 1) face(x, y, p.nz);
}

__global__ void __launch_bounds__(128) cfgAdvectVelocity(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                         Velocity vel, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= p.nx) return;
    facesOfCell(p, x, blockIdx.y, blockIdx.z, [&](int fx, int fy, int fz) { cfgAdvectVelocityAt(uOut, vOut, wOut, vel, p, fx, fy, fz); });
}

// Backtrace of record a from the cell centre, then burn, decay and emitters.
__device__ __forceinline__ void cfgAdvectScalarsAt(Rec4* __restrict__ aOut, const Rec4* __restrict__ aIn, const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    const float px = static_cast<float>(x) + 0.5f, py = static_cast<float>(y) + 0.5f, pz = static_cast<float>(z) + 0.5f;
    const float3 d = velocityAtCentre(vel, p, x, y, z);
    const float4 s = recordAt(aIn, p, px - d.x, py - d.y, pz - d.z);
    float heat = s.x, fuel = s.y, soot = s.w;
    if (heat > p.ignition) {
        const float burn = fuel * p.burnFrac;
        fuel = fuel - burn;
        heat = heat + p.heatRelease * burn;
        soot = soot + p.sootYield * burn;
    }
    heat = heat - heat * p.coolFrac;
    soot = soot - soot * p.sootFrac;
    const unsigned cell = static_cast<unsigned>((z * p.ny + y) * p.nx + x);
    for (int e = 0; e < p.emitterCount; ++e) {
        const ConfigEmitter& em = p.emitters[e];
        if (!inDisk(em, x, y, z)) continue;
        const float j = 1.0f - em.jitter * jitterUniform(em.seed, p.step, cell);
        fuel = fmaxf(fuel, em.fuel * j);
        heat = fmaxf(heat, em.heat * j);
    }
    stv(aOut + cell, make_float4(heat, fuel, 0.0f, soot));
}

__global__ void __launch_bounds__(128) cfgAdvectScalars(Rec4* __restrict__ aOut, const Rec4* __restrict__ aIn, Velocity vel, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= p.nx) return;
    cfgAdvectScalarsAt(aOut, aIn, vel, p, x, y, z);
}

// omega = curl of the cell-centred velocity (central differences, clamped
// neighbours), and |omega|.
__device__ __forceinline__ void cfgVorticityAt(float4* __restrict__ vort, const Velocity& vel, const ConfigParams& p, int x, int y, int z) {
    const int xm = max(x - 1, 0), xp = min(x + 1, p.nx - 1);
    const int ym = max(y - 1, 0), yp = min(y + 1, p.ny - 1);
    const int zm = max(z - 1, 0), zp = min(z + 1, p.nz - 1);
    const int ux = p.nx + 1, vy = p.ny + 1;
    auto ccx = [&](int i, int j, int k) { return cellCentred(vel.u, faceIndex(i, j, k, ux, p.ny), faceIndex(i + 1, j, k, ux, p.ny)); };
    auto ccy = [&](int i, int j, int k) { return cellCentred(vel.v, faceIndex(i, j, k, p.nx, vy), faceIndex(i, j + 1, k, p.nx, vy)); };
    auto ccz = [&](int i, int j, int k) { return cellCentred(vel.w, faceIndex(i, j, k, p.nx, p.ny), faceIndex(i, j, k + 1, p.nx, p.ny)); };
    const float ox = 0.5f * (ccz(x, yp, z) - ccz(x, ym, z)) - 0.5f * (ccy(x, y, zp) - ccy(x, y, zm));
    const float oy = 0.5f * (ccx(x, y, zp) - ccx(x, y, zm)) - 0.5f * (ccz(xp, y, z) - ccz(xm, y, z));
    const float oz = 0.5f * (ccy(xp, y, z) - ccy(xm, y, z)) - 0.5f * (ccx(x, yp, z) - ccx(x, ym, z));
    vort[(z * p.ny + y) * p.nx + x] = make_float4(ox, oy, oz, sqrtf(ox * ox + oy * oy + oz * oz));
}

__global__ void __launch_bounds__(128) cfgVorticity(float4* __restrict__ vort, Velocity vel, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= p.nx) return;
    cfgVorticityAt(vort, vel, p, x, y, z);
}

// The curl-noise acceleration amplitude * curl(psi) at every cell centre.  It
// depends only on the noise parameters and the grid, so the scene builds it
// once per parameter set and cfgCellForce reads it.
__device__ __forceinline__ void cfgNoiseFieldAt(float4* __restrict__ noise, const ConfigParams& p, int x, int y, int z) {
    const float px = static_cast<float>(x) + 0.5f, py = static_cast<float>(y) + 0.5f, pz = static_cast<float>(z) + 0.5f;
    const float3 g0 = noiseGradient(p, 0, px, py, pz);
    const float3 g1 = noiseGradient(p, 1, px, py, pz);
    const float3 g2 = noiseGradient(p, 2, px, py, pz);
    noise[(z * p.ny + y) * p.nx + x] = make_float4(p.noiseAmp * (g2.y - g1.z), p.noiseAmp * (g0.z - g2.x), p.noiseAmp * (g1.x - g0.y), 0.0f);
}

__global__ void __launch_bounds__(128) cfgNoiseField(float4* __restrict__ noise, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= p.nx) return;
    cfgNoiseFieldAt(noise, p, x, y, z);
}

// Cell-centred acceleration: buoyancy + confinement + curl noise (read from
// the field cfgNoiseField built; null when the amplitude is 0).
__device__ __forceinline__ void cfgCellForceAt(float4* __restrict__ force, const float4* __restrict__ vort, const Rec4* __restrict__ a,
                                                    const float4* __restrict__ noise, const ConfigParams& p, int x, int y, int z) {
    const int idx = (z * p.ny + y) * p.nx + x;
    const float4 s = ldv(a + idx);
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    if (p.eps != 0.0f) {
        const int xm = max(x - 1, 0), xp = min(x + 1, p.nx - 1);
        const int ym = max(y - 1, 0), yp = min(y + 1, p.ny - 1);
        const int zm = max(z - 1, 0), zp = min(z + 1, p.nz - 1);
        const float4 o = vort[idx];
        const float ex = 0.5f * (vort[(z * p.ny + y) * p.nx + xp].w - vort[(z * p.ny + y) * p.nx + xm].w);
        const float ey = 0.5f * (vort[(z * p.ny + yp) * p.nx + x].w - vort[(z * p.ny + ym) * p.nx + x].w);
        const float ez = 0.5f * (vort[(zp * p.ny + y) * p.nx + x].w - vort[(zm * p.ny + y) * p.nx + x].w);
        const float len = sqrtf(ex * ex + ey * ey + ez * ez);
        float nx = 0.0f, ny = 0.0f, nz = 0.0f;
        if (len > 1e-20f) {
            nx = ex / len;
            ny = ey / len;
            nz = ez / len;
        }
        cx = p.eps * (ny * o.z - nz * o.y);
        cy = p.eps * (nz * o.x - nx * o.z);
        cz = p.eps * (nx * o.y - ny * o.x);
    }
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    if (p.noiseAmp != 0.0f) {
        const float4 n = __ldg(noise + idx);
        fx = n.x;
        fy = n.y;
        fz = n.z;
    }
    const float buoyancy = p.buoyHeat * (s.x - p.ambient) - p.buoySoot * s.w;
    force[idx] = make_float4(cx + fx, buoyancy + cy + fy, cz + fz, 0.0f);
}

__global__ void __launch_bounds__(128) cfgCellForce(float4* __restrict__ force, const float4* __restrict__ vort, const Rec4* __restrict__ a,
                                                    const float4* __restrict__ noise, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= p.nx) return;
    cfgCellForceAt(force, vort, a, noise, p, x, y, z);
}

// Faces += dt * (mean of the two adjacent cells' accelerations) + wind; the
// emitter cells' v faces take upVelocity; walls (u at x = 0, nx; v at y = 0;
// w at z = 0, nz) are zero; the top v faces keep the cell below's acceleration.
__device__ __forceinline__ void cfgApplyForcesAt(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                      const Velocity& vel, const float4* __restrict__ force, const ConfigParams& p, int x, int y, int z) {
    if (y < p.ny && z < p.nz) {
        const int i = faceIndex(x, y, z, p.nx + 1, p.ny);
        float u = 0.0f;
        if (x > 0 && x < p.nx) {
            const float fa = force[(z * p.ny + y) * p.nx + x - 1].x, fb = force[(z * p.ny + y) * p.nx + x].x;
            u = ldv(vel.u + i) + (p.dt * (0.5f * (fa + fb)) + p.windDtX);
        }
        stv(uOut + i, u);
    }
    if (x < p.nx && z < p.nz) {
        const int i = faceIndex(x, y, z, p.nx, p.ny + 1);
        float v = 0.0f;
        if (y > 0) {
            const float fd = force[(z * p.ny + y - 1) * p.nx + x].y;
            v = y < p.ny ? ldv(vel.v + i) + p.dt * (0.5f * (fd + force[(z * p.ny + y) * p.nx + x].y)) : ldv(vel.v + i) + p.dt * fd;
            for (int e = 0; e < p.emitterCount; ++e) {
                const ConfigEmitter& em = p.emitters[e];
                if ((y < p.ny && inDisk(em, x, y, z)) || inDisk(em, x, y - 1, z)) v = em.up;
            }
        }
        stv(vOut + i, v);
    }
    if (x < p.nx && y < p.ny) {
        const int i = faceIndex(x, y, z, p.nx, p.ny);
        float w = 0.0f;
        if (z > 0 && z < p.nz) {
            const float fb = force[((z - 1) * p.ny + y) * p.nx + x].z, ff = force[(z * p.ny + y) * p.nx + x].z;
            w = ldv(vel.w + i) + (p.dt * (0.5f * (fb + ff)) + p.windDtZ);
        }
        stv(wOut + i, w);
    }
}

__global__ void __launch_bounds__(128) cfgApplyForces(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                      Velocity vel, const float4* __restrict__ force, ConfigParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= p.nx) return;
    facesOfCell(p, x, blockIdx.y, blockIdx.z,
                [&](int fx, int fy, int fz) { cfgApplyForcesAt(uOut, vOut, wOut, vel, force, p, fx, fy, fz); });
}

// ---- empty space ------------------------------------------------------------
// A fire and its smoke fill part of the grid (0.6% of 128^3 after 10 steps, 13%
// after 60; 40% of 64^3 after 40), and a sample of cells where heat, fuel and
// soot are all zero leaves the light's tau and the pixel's sums as they are, to
// the bit: its extinction is 0 (of either sign), its alpha 1 - exp(0) = 0, and 0
// is added to sums that start at +0.  So samples are evaluated where a brick of
// 4x4x4 cells holds something (CfgOccupancy): a ray's samples are cut to the set
// bricks' bounding box, widened by more than the rounding of the positions, and
// in it a sample's first corner, computed as the sample computes it, tells its
// brick.  The exceptions: a step, a light colour or a transmittance so large that
// 0 times it could be NaN evaluates every sample, and so does a pixel whose
// remaining view is infinite or NaN, from there on.  Where half of the bricks are
// set, only the cut to the box is made, and a grid that is largely full (48 of 64
// cells spread over it) takes every sample: its records are not read, and the
// kernels run the plain loop, whose samples overlap better than the cut one's
// (full 192^3, 65,536 rays of one lane: 213 us in the cut loop, 136 in the plain
// one).  Measured (light, render, each with its build): 128^3 after 40 steps 138 ->
// 31 and 440 -> 95 us, 256^3 1014 -> 86 and 486 -> 138 us; full grids, in sum, 128^3
// 561 and 557 us, 256^3 1493 and 1500, 64^3 159 and 131.  The build takes 4 us on a
// full grid, 10 at 128^3 and 65 at 256^3 otherwise (floor 41: the record once).

__device__ __forceinline__ bool seen(float4 r) { return (r.x != 0.0f) | (r.y != 0.0f) | (r.w != 0.0f); }

// One warp's share of the build: the units (cfgOccupancyUnits) warp, warp + warps,
// ...; tr: also checks that every transmittance is regular.  Bound by its reads
// of record a, (5/4)^2 of them through L2: a warp keeps the box and the count of
// its units in registers, as the atomics of every unit took as long as the reads.
// The last warp to finish publishes the box and clears the accumulators for the
// next build.
__device__ __forceinline__ void cfgOccupancyAt(CfgOccupancy* occ, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                               const ConfigParams& p, int warp, int warps, int lane) {
    const int bx = cfgBricks(p.nx), by = cfgBricks(p.ny), bz = cfgBricks(p.nz);
    const int perRow = (bx + 6) / 7;
    const int units = perRow * by * bz;
    // Every warp looks at the same cells of the same records, so all take the same way.
    int full = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int x = (2 * (lane & 3) + 1) * p.nx / 8, y = (2 * ((lane >> 2) & 3) + 1) * p.ny / 8, z = (2 * (2 * k + (lane >> 4)) + 1) * p.nz / 8;
        full += __popc(__ballot_sync(0xffffffffu, seen(ldv(a + faceIndex(x, y, z, p.nx, p.ny)))));
    }
    if (full >= 48) {
        if (warp == 0 && lane == 0) occ->look = kCfgEvery;
        return;
    }
    unsigned lo = 0u, hi = 0u, count = 0u;  // the set bricks' ends in the axis lane % 3, and their number
    for (int unit = warp; unit < units; unit += warps) {
        const int row = unit / perRow, chunk = unit - row * perRow;
        const int Z = row / by, Y = row - Z * by;
        const int x = min(28 * chunk + lane, p.nx - 1);
        // Past the grid's ends the last cell again; all 25 loads in flight.
        bool any = false;  // (|, not ||: a short circuit would wait for each load)
#pragma unroll
        for (int dz = 0; dz < 5; ++dz) {
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) any |= seen(ldv(a + faceIndex(x, min(4 * Y + dy, p.ny - 1), min(4 * Z + dz, p.nz - 1), p.nx, p.ny)));
        }
        const unsigned cells = __ballot_sync(0xffffffffu, any);
        const int X = 7 * chunk + lane;
        bool set = false;
        if (lane < 7 && X < bx) {
            set = ((cells >> (4 * lane)) & 31u) != 0u;
            reinterpret_cast<unsigned char*>(occ + 1)[(Z * by + Y) * bx + X] = set ? 1 : 0;
        }
        const unsigned f = __ballot_sync(0xffffffffu, set);
        if (f == 0u) continue;
        count += static_cast<unsigned>(__popc(f));
        const int axis = lane % 3;
        const int first = axis == 0 ? 7 * chunk + __ffs(static_cast<int>(f)) - 1 : axis == 1 ? Y : Z;
        const int last = axis == 0 ? 7 * chunk + 31 - __clz(static_cast<int>(f)) : axis == 1 ? Y : Z;
        lo = max(lo, (1u << 20) - static_cast<unsigned>(first));
        hi = max(hi, static_cast<unsigned>(last) + 1u);
    }
    bool irregular = false;
    if (tr != nullptr) {
        const int n = p.lx * p.ly * p.lz;
        for (int i = warp * 32 + lane; i < n; i += min(warps, units) * 32) irregular = irregular || !(fabsf(__ldg(tr + i)) <= 1e30f);
    }
    irregular = __any_sync(0xffffffffu, irregular);
    // Lanes 0-2 the box's low ends, 3-5 its high ends.
    if (lane == 7 && count != 0u) atomicAdd(&occ->accSet, count);
    if (lane < 6 && count != 0u) atomicMax(&occ->acc[lane], lane < 3 ? lo : hi);
    if (irregular && lane == 6) atomicOr(&occ->accIrregular, 1u);
    __threadfence();
    __syncwarp();
    const unsigned participants = static_cast<unsigned>(min(warps, units));
    unsigned done = 0u;
    if (lane == 0) done = atomicInc(&occ->done, participants - 1u);  // wraps to 0 for the next build
    if (__shfl_sync(0xffffffffu, done, 0) != participants - 1u) return;
    __threadfence();
    if (lane < 6) occ->box[lane] = atomicExch(&occ->acc[lane], 0u);
    if (lane == 6) occ->irregular = atomicExch(&occ->accIrregular, 0u);
    // Set bricks in half the grid or more: asking for each sample costs more than it saves.
    if (lane == 7) {
        const unsigned bricks = static_cast<unsigned>(bx) * static_cast<unsigned>(by) * static_cast<unsigned>(bz);
        occ->look = atomicExch(&occ->accSet, 0u) >= bricks / 2u ? kCfgBox : kCfgAsk;
    }
}

__global__ void __launch_bounds__(128) cfgOccupancyBuild(CfgOccupancy* occ, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                                         ConfigParams p) {
    const int warp = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (warp >= cfgOccupancyUnits(p.nx, p.ny, p.nz)) return;
    cfgOccupancyAt(occ, a, tr, p, warp, gridDim.x * 4, threadIdx.x & 31);
}

// The samples first .. last - 1 of a ray (origin + direction * (t0 + (s + 0.5)
// ds), s = 0 .. count - 1, in cells) that may lie in the bricks' box.
__device__ __forceinline__ void samplesInBox(const CfgOccupancy* occ, const ConfigParams& p, const float (&origin)[3], const float (&dir)[3],
                                             float t0, float ds, int count, int& first, int& last) {
    const int bricks[3] = {cfgBricks(p.nx), cfgBricks(p.ny), cfgBricks(p.nz)};
    // Past the rounding of the positions (a few ulp of their terms).
    const float margin = 0.25f + 1e-6f * (fabsf(origin[0]) + fabsf(origin[1]) + fabsf(origin[2]) + t0 + static_cast<float>(count) * ds);
    float from = -3.0e38f, to = 3.0e38f;
    bool hit = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int lo = (1 << 20) - static_cast<int>(occ->box[k]), hi = static_cast<int>(occ->box[3 + k]) - 1;
        if (hi < 0) hit = false;
        // Positions past the grid's ends are clamped to its first and last cells.
        const float a = lo == 0 ? -3.0e38f : static_cast<float>(4 * lo) + 0.5f - margin;
        const float b = hi == bricks[k] - 1 ? 3.0e38f : static_cast<float>(4 * hi) + 4.5f + margin;
        if (dir[k] == 0.0f) {
            if (origin[k] < a || origin[k] > b) hit = false;
        } else {
            const float ta = (a - origin[k]) / dir[k], tb = (b - origin[k]) / dir[k];
            from = fmaxf(from, fminf(ta, tb));
            to = fminf(to, fmaxf(ta, tb));
        }
    }
    first = last = 0;
    if (!hit || from > to) return;
    last = count;
    if (ds > 1e-20f) {
        const float n = static_cast<float>(count);
        first = static_cast<int>(fminf(fmaxf((from - t0) / ds - 2.0f, 0.0f), n));
        last = static_cast<int>(fminf(fmaxf((to - t0) / ds + 2.0f, 0.0f), n));
    }
}

// Rays are taken by a lane each or, where that leaves the chip short of warps
// (kLightLaneRays, pixelLanes), by kRayLanes lanes each: a lane evaluates every kRayLanes-th
// sample, and all of them add the samples' terms in order, passed by shuffles,
// so the sums are the same to the bit.  sub is the lane's number in its ray; the
// warp's rays walk their samples together, full warps only.

// Whether a lane that walks along has its flag set: this one, or (LANES > 1) any
// of the warp's.
template <int LANES>
__device__ __forceinline__ bool anyOf(bool own) {
    if constexpr (LANES == 1) {
        return own;
    } else {
        return __any_sync(0xffffffffu, own) != 0;
    }
}
// The sample range to walk: this ray's, or the least one that has the warp's.
template <int LANES>
__device__ __forceinline__ void widen(int& first, int& last) {
    if constexpr (LANES > 1) {
        first = __reduce_min_sync(0xffffffffu, first);
        last = __reduce_max_sync(0xffffffffu, last);
    }
}
// Value v of lane j of the ray.
template <int LANES>
__device__ __forceinline__ float fromLane(float v, int j) {
    if constexpr (LANES == 1) {
        return v;
    } else {
        return __shfl_sync(0xffffffffu, v, j, LANES);
    }
}

// Transmittance toward the point light from the centre of each 2x2x2 block of
// cells: lightSamples midpoint samples of extinction * S + fuelExtinction * F
// along the segment, clipped where it leaves the grid box.
// SKIP: with an occupancy, else every sample.  BESIDE: compiled beside the form
// with one, where the plain loop of a kernel of its own came out slower (full
// 128^3 181 us instead of 144).
template <int LANES, bool SKIP, bool BESIDE = false>
__device__ __forceinline__ void cfgTransmittanceAt(float* __restrict__ tr, const Rec4* __restrict__ a, CfgOccupancy* occ, const ConfigParams& p,
                                                   int lx, int ly, int lz, int sub, bool live) {
    const float px = 2.0f * static_cast<float>(lx) + 1.0f, py = 2.0f * static_cast<float>(ly) + 1.0f, pz = 2.0f * static_cast<float>(lz) + 1.0f;
    const float dx = p.light.x - px, dy = p.light.y - py, dz = p.light.z - pz;
    const float dist = sqrtf(dx * dx + dy * dy + dz * dz);
    const bool apart = dist > 1e-6f;
    const float rx = dx / dist, ry = dy / dist, rz = dz / dist;
    float seg = dist;
    if (rx > 0.0f) seg = fminf(seg, (static_cast<float>(p.nx) - px) / rx);
    if (rx < 0.0f) seg = fminf(seg, (0.0f - px) / rx);
    if (ry > 0.0f) seg = fminf(seg, (static_cast<float>(p.ny) - py) / ry);
    if (ry < 0.0f) seg = fminf(seg, (0.0f - py) / ry);
    if (rz > 0.0f) seg = fminf(seg, (static_cast<float>(p.nz) - pz) / rz);
    if (rz < 0.0f) seg = fminf(seg, (0.0f - pz) / rz);
    seg = fmaxf(seg, 0.0f);
    const float ds = seg / static_cast<float>(p.lightSamples);
    float tau = 0.0f;
    if constexpr (LANES == 1 && !SKIP && !BESIDE) {
        if (apart) {
            for (int s = 0; s < p.lightSamples; ++s) {
                const float at = (static_cast<float>(s) + 0.5f) * ds;
                const float4 r = recordAt(a, p, px + rx * at, py + ry * at, pz + rz * at);
                tau = tau + (p.extinction * r.w + p.fuelExtinction * r.y) * ds;
            }
        }
    } else {
        const unsigned look = SKIP ? occ->look : static_cast<unsigned>(kCfgEvery);
        const bool skip = look != kCfgEvery && ds < 1e30f, ask = skip && look == kCfgAsk;
        int first = 0, last = p.lightSamples;
        if (skip) {
            const float origin[3] = {px, py, pz}, dir[3] = {rx, ry, rz};
            samplesInBox(occ, p, origin, dir, 0.0f, ds, p.lightSamples, first, last);
        }
        if (!apart || !live) first = last = 0;
        const int bx = cfgBricks(p.nx), by = cfgBricks(p.ny);
        int from = last > first ? first : p.lightSamples, to = last;
        widen<LANES>(from, to);
        if (LANES == 1 && !ask) {  // no branch in the loop, so that samples overlap
            for (int s = first; s < last; ++s) {
                const float at = (static_cast<float>(s) + 0.5f) * ds;
                const float4 r = recordAt(a, p, px + rx * at, py + ry * at, pz + rz * at);
                tau = tau + (p.extinction * r.w + p.fuelExtinction * r.y) * ds;
            }
            to = from;
        }
        for (int s0 = from; s0 < to; s0 += LANES) {
            const int s = s0 + sub;
            const float at = (static_cast<float>(s) + 0.5f) * ds;
            const auto c = recordCorners(p, px + rx * at, py + ry * at, pz + rz * at);
            bool own = s >= first && s < last;
            if (own && ask) own = brickSeen(occ, c, bx, by);
            if (!anyOf<LANES>(own)) continue;
            float term = 0.0f;
            if (own) {
                const float4 r = trilinearRec(a, c, p.nx, p.ny);
                term = (p.extinction * r.w + p.fuelExtinction * r.y) * ds;
            }
#pragma unroll
            for (int j = 0; j < LANES; ++j) tau = tau + fromLane<LANES>(term, j);
        }
    }
    if (!live || sub != 0) return;
    const float t = apart ? expf(-tau) : 1.0f;
    tr[(lz * p.ly + ly) * p.lx + lx] = t;
    if (SKIP && !(fabsf(t) <= 1e30f)) occ->irregular = 1u;
}

template <bool SKIP>
__device__ __forceinline__ void cfgTransmittanceOwn(float* __restrict__ tr, const Rec4* __restrict__ a, CfgOccupancy* occ, const ConfigParams& p) {
    const int lx = blockIdx.x * blockDim.x + threadIdx.x;
    const int ly = blockIdx.y;
    const int lz = blockIdx.z;
    if (lx >= p.lx) return;
    if (SKIP && occ->look == kCfgEvery) {  // (a copy of its own: in one loop with the cut the registers slow both)
        cfgTransmittanceAt<1, false, true>(tr, a, occ, p, lx, ly, lz, 0, true);
        return;
    }
    cfgTransmittanceAt<1, SKIP>(tr, a, occ, p, lx, ly, lz, 0, true);
}
template <bool SKIP>
__device__ __forceinline__ void cfgTransmittanceShared(float* __restrict__ tr, const Rec4* __restrict__ a, CfgOccupancy* occ,
                                                       const ConfigParams& p) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kRayLanes, row = i / p.lx;
    cfgTransmittanceAt<kRayLanes, SKIP>(tr, a, occ, p, i - row * p.lx, row % p.ly, row / p.ly, threadIdx.x % kRayLanes,
                                        i < p.lx * p.ly * p.lz);
}
__global__ void __launch_bounds__(128) cfgTransmittance(float* __restrict__ tr, const Rec4* __restrict__ a, CfgOccupancy* occ, ConfigParams p) {
    cfgTransmittanceOwn<true>(tr, a, occ, p);
}
__global__ void __launch_bounds__(128) cfgTransmittanceEvery(float* __restrict__ tr, const Rec4* __restrict__ a, ConfigParams p) {
    cfgTransmittanceOwn<false>(tr, a, nullptr, p);
}
__global__ void __launch_bounds__(128) cfgTransmittanceLanes(float* __restrict__ tr, const Rec4* __restrict__ a, CfgOccupancy* occ,
                                                             ConfigParams p) {
    cfgTransmittanceShared<true>(tr, a, occ, p);
}
__global__ void __launch_bounds__(128) cfgTransmittanceLanesEvery(float* __restrict__ tr, const Rec4* __restrict__ a, ConfigParams p) {
    cfgTransmittanceShared<false>(tr, a, nullptr, p);
}

// One pixel: the camera ray's chord through the grid box in primarySamples
// midpoint samples; absorption, in-scattering of the point light (its
// transmittance volume) and emission; a dark background behind.
template <int LANES, bool SKIP>
__device__ __forceinline__ void cfgRaymarchAt(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                              const CfgOccupancy* __restrict__ occ, const ConfigParams& p, int px, int py, int sub, bool live) {
    const float sx = (2.0f * (static_cast<float>(px) + 0.5f) / static_cast<float>(p.frameW) - 1.0f) * p.tanHalf * p.aspect;
    const float sy = (1.0f - 2.0f * (static_cast<float>(py) + 0.5f) / static_cast<float>(p.frameH)) * p.tanHalf;
    float dx = p.forward.x + p.right.x * sx + p.up.x * sy;
    float dy = p.forward.y + p.right.y * sx + p.up.y * sy;
    float dz = p.forward.z + p.right.z * sx + p.up.z * sy;
    const float len = sqrtf(dx * dx + dy * dy + dz * dz);
    dx = dx / len;
    dy = dy / len;
    dz = dz / len;
    float t0 = 0.0f, t1 = 3.0e38f;
    bool hit = live;
    const float eye[3] = {p.eye.x, p.eye.y, p.eye.z};
    const float dir[3] = {dx, dy, dz};
    const float hiB[3] = {static_cast<float>(p.nx), static_cast<float>(p.ny), static_cast<float>(p.nz)};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (dir[k] == 0.0f) {
            if (eye[k] < 0.0f || eye[k] > hiB[k]) hit = false;
        } else {
            const float ta = (0.0f - eye[k]) / dir[k];
            const float tb = (hiB[k] - eye[k]) / dir[k];
            t0 = fmaxf(t0, fminf(ta, tb));
            t1 = fminf(t1, fmaxf(ta, tb));
        }
    }
    float r = 0.0f, g = 0.0f, b = 0.0f, view = 1.0f;
    const float ds = (t1 - t0) / static_cast<float>(p.primarySamples);
    const unsigned look = SKIP ? occ->look : static_cast<unsigned>(kCfgEvery);
    const bool skip = look != kCfgEvery && ds < 1e30f && fabsf(p.albedo * p.lightIntensity) <= 1e8f && (!SKIP || occ->irregular == 0u);
    const bool ask = skip && look == kCfgAsk;
    int first = 0, last = p.primarySamples;
    if (skip) samplesInBox(occ, p, eye, dir, t0, ds, p.primarySamples, first, last);
    hit = hit && t1 > t0;
    if (!hit) first = last = 0;
    const int bx = cfgBricks(p.nx), by = cfgBricks(p.ny);
    int from = last > first ? first : p.primarySamples, to = last;
    widen<LANES>(from, to);
    float termR, termG, termB, through;
    auto evaluate = [&](int s) {
        const float at = t0 + (static_cast<float>(s) + 0.5f) * ds;
        const float qx = p.eye.x + dx * at, qy = p.eye.y + dy * at, qz = p.eye.z + dz * at;
        const float4 rec = recordAt(a, p, qx, qy, qz);
        const float sigma = p.extinction * rec.w + p.fuelExtinction * rec.y;
        const float alpha = 1.0f - expf(-(sigma * ds));
        const float lt = trilinear1(tr, cornersAt(qx * 0.5f - 0.5f, qy * 0.5f - 0.5f, qz * 0.5f - 0.5f, p.lx, p.ly, p.lz), p.lx, p.ly);
        const float scatter = p.albedo * p.lightIntensity * lt * alpha;
        const float heat = fmaxf(rec.x, 0.0f);
        const float h = heat / (heat + 1.0f);
        const float e = p.emission * heat * ds;
        termR = scatter + e;
        termG = scatter + e * (0.35f + 0.45f * h);
        termB = scatter + e * (0.08f + 0.50f * h * h);
        through = 1.0f - alpha;
    };
    auto add = [&](int j) {
        r = r + view * fromLane<LANES>(termR, j);
        g = g + view * fromLane<LANES>(termG, j);
        b = b + view * fromLane<LANES>(termB, j);
        view = view * fromLane<LANES>(through, j);
    };
    if (LANES == 1 && !ask) {  // no branch in the loop, so that samples overlap
        for (int s = first; s < last; ++s) {
            evaluate(s);
            add(0);
        }
        to = from;
    }
    for (int s0 = from; s0 < to; s0 += LANES) {
        const int s = s0 + sub;
        const float at = t0 + (static_cast<float>(s) + 0.5f) * ds;
        bool own = s >= first && s < last;
        // (0 times a view that is infinite or NaN is NaN: then every sample counts.)
        if (own && ask) {
            own = brickSeen(occ, recordCorners(p, p.eye.x + dx * at, p.eye.y + dy * at, p.eye.z + dz * at), bx, by) || !(fabsf(view) <= 3.0e38f);
        }
        if (!anyOf<LANES>(own)) continue;
        termR = termG = termB = 0.0f;
        through = 1.0f;
        if (own) evaluate(s);
        // The ray's own samples only: 0 times an infinite view would be NaN.
#pragma unroll
        for (int j = 0; j < LANES; ++j) {
            if (LANES == 1 || s0 + j < p.primarySamples) add(j);
        }
    }
    if (!live || sub != 0) return;
    if (hit && last < p.primarySamples) {  // the samples after the last one add 0 times the view
        r = r + view * 0.0f;
        g = g + view * 0.0f;
        b = b + view * 0.0f;
    }
    hdr[py * p.frameW + px] = make_float4(r + view * 0.015f, g + view * 0.016f, b + view * 0.020f, 1.0f - view);
}

template <bool SKIP>
__device__ __forceinline__ void cfgRaymarchOwn(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                               const CfgOccupancy* __restrict__ occ, const ConfigParams& p) {
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= p.frameW || py >= p.frameH) return;
    if (SKIP && occ->look == kCfgEvery) {
        cfgRaymarchAt<1, false>(hdr, a, tr, occ, p, px, py, 0, true);
        return;
    }
    cfgRaymarchAt<1, SKIP>(hdr, a, tr, occ, p, px, py, 0, true);
}
// A warp's rays are 4 x 2 pixels, a block's 16 x 2.
template <bool SKIP>
__device__ __forceinline__ void cfgRaymarchShared(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                                  const CfgOccupancy* __restrict__ occ, const ConfigParams& p) {
    const int ray = (threadIdx.x & 31) / kRayLanes, warp = threadIdx.x >> 5;
    const int px = blockIdx.x * 16 + warp * 4 + (ray & 3);
    const int py = blockIdx.y * 2 + (ray >> 2);
    cfgRaymarchAt<kRayLanes, SKIP>(hdr, a, tr, occ, p, px, py, threadIdx.x % kRayLanes, px < p.frameW && py < p.frameH);
}
__global__ void __launch_bounds__(128) cfgRaymarch(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                                   const CfgOccupancy* __restrict__ occ, ConfigParams p) {
    cfgRaymarchOwn<true>(hdr, a, tr, occ, p);
}
__global__ void __launch_bounds__(128) cfgRaymarchEvery(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                                        ConfigParams p) {
    cfgRaymarchOwn<false>(hdr, a, tr, nullptr, p);
}
__global__ void __launch_bounds__(128) cfgRaymarchLanes(float4* __restrict__ hdr, const Rec4* __restrict__ a, const float* __restrict__ tr,
                                                        const CfgOccupancy* __restrict__ occ, ConfigParams p) {
    cfgRaymarchShared<true>(hdr, a, tr, occ, p);
}
__global__ void __launch_bounds__(128) cfgRaymarchLanesEvery(float4* __restrict__ hdr, const Rec4* __restrict__ a,
                                                             const float* __restrict__ tr, ConfigParams p) {
    cfgRaymarchShared<false>(hdr, a, tr, nullptr, p);
}

// ---- the incremental projection of the multigrid solve (fire_mg.cu) ----

// The incremental projection's first half (see the file comment), out of
// place: per cell, the faces it owns (u at x, v at y, w at z, and the last
// face of each axis for the last cell) are written to the other velocity
// buffer, the interior ones and the top ones minus the previous pressure's
// gradient, rounded to storage, the wall ones as they are; rhs = -div of the
// cell's six updated faces (those it does not own recomputed the same way).
__device__ __forceinline__ void cfgPrepareIncrementAt(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                      const Velocity& vel, const float* __restrict__ pressure, float* __restrict__ rhs,
                                                      int nx, int ny, int nz, int x, int y, int z) {
    const int i = (z * ny + y) * nx + x;
    const int ui = (z * ny + y) * (nx + 1) + x;
    const int vi = (z * (ny + 1) + y) * nx + x;
    const int wi = (z * ny + y) * nx + x;
    const float pc = pressure[i];
    const float u0 = x > 0 ? storageRound(ldv(vel.u + ui) - (pc - pressure[i - 1])) : ldv(vel.u + ui);
    const float u1 = x + 1 < nx ? storageRound(ldv(vel.u + ui + 1) - (pressure[i + 1] - pc)) : ldv(vel.u + ui + 1);
    const float v0 = y > 0 ? storageRound(ldv(vel.v + vi) - (pc - pressure[i - nx])) : ldv(vel.v + vi);
    const float v1 = y + 1 < ny ? storageRound(ldv(vel.v + vi + nx) - (pressure[i + nx] - pc))
                                : storageRound(ldv(vel.v + vi + nx) - ((0.0f - pc) - pc));
    const float w0 = z > 0 ? storageRound(ldv(vel.w + wi) - (pc - pressure[i - nx * ny])) : ldv(vel.w + wi);
    const float w1 = z + 1 < nz ? storageRound(ldv(vel.w + wi + nx * ny) - (pressure[i + nx * ny] - pc)) : ldv(vel.w + wi + nx * ny);
    const float div = u1 - u0 + v1 - v0 + w1 - w0;
    rhs[i] = -div;
    stv(uOut + ui, u0);
    stv(vOut + vi, v0);
    stv(wOut + wi, w0);
    if (x == nx - 1) stv(uOut + ui + 1, u1);
    if (y == ny - 1) stv(vOut + vi + nx, v1);
    if (z == nz - 1) stv(wOut + wi + nx * ny, w1);
}

// The incremental projection's second half: u -= grad delta on the interior
// faces and the top faces (ghost -delta); with doWalls the closed walls are
// zeroed as in subtractWall.
__device__ __forceinline__ void cfgSubtractIncrementAt(FaceT* __restrict__ u, FaceT* __restrict__ v, FaceT* __restrict__ w,
                                                       const float* __restrict__ delta, int nx, int ny, int nz, int doWalls, int x, int y,
                                                       int z) {
    const int i = (z * ny + y) * nx + x;
    const float dc = delta[i];
    const int ui = (z * ny + y) * (nx + 1) + x;
    const int vi = (z * (ny + 1) + y) * nx + x;
    const int wi = (z * ny + y) * nx + x;
    if (x > 0) stv(u + ui, ldv(u + ui) - (dc - delta[i - 1]));
    if (y > 0) stv(v + vi, ldv(v + vi) - (dc - delta[i - nx]));
    if (z > 0) stv(w + wi, ldv(w + wi) - (dc - delta[i - nx * ny]));
    if (y == ny - 1) {
        const int top = (z * (ny + 1) + ny) * nx + x;
        stv(v + top, ldv(v + top) - ((0.0f - dc) - dc));
    }
    if (doWalls) {
        if (x == 0) stv(u + ui, 0.0f);
        if (x == nx - 1) stv(u + ui + 1, 0.0f);
        if (y == 0) stv(v + vi, 0.0f);
        if (z == 0) stv(w + wi, 0.0f);
        if (z == nz - 1) stv(w + (nz * ny + y) * nx + x, 0.0f);
    }
}

__global__ void __launch_bounds__(128) cfgPrepareIncrement(FaceT* __restrict__ uOut, FaceT* __restrict__ vOut, FaceT* __restrict__ wOut,
                                                           Velocity vel, const float* __restrict__ pressure, float* __restrict__ rhs,
                                                           int nx, int ny, int nz) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= nx) return;
    cfgPrepareIncrementAt(uOut, vOut, wOut, vel, pressure, rhs, nx, ny, nz, x, blockIdx.y, blockIdx.z);
}

__global__ void __launch_bounds__(128) cfgSubtractIncrement(FaceT* __restrict__ u, FaceT* __restrict__ v, FaceT* __restrict__ w,
                                                            const float* __restrict__ delta, int nx, int ny, int nz, int doWalls) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= nx) return;
    cfgSubtractIncrementAt(u, v, w, delta, nx, ny, nz, doWalls, x, blockIdx.y, blockIdx.z);
}

// ---- batched stages (BatchScene, BatchPlan in fire_kernels.h) ----------

namespace {

// The scene of this block: the last s with start[s] <= blockIdx.x.
__device__ __forceinline__ int batchSceneOf(const int* start, int n) {
    const int b = static_cast<int>(blockIdx.x);
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(start + mid) <= b) {
            lo = mid;
        } else {
            hi = mid;
        }
    }
    return lo;
}

// This thread's batchPerThread(space) elements of index space `space`, in
// rows of w elements and planes of h rows: body(B, i, x, y, z) for each.  A
// block takes kBatchThreads * K consecutive elements and thread t the
// elements t, t + kBatchThreads, ... of them (so that every pass of the
// block is coalesced); the scene lookup and the division of the first index
// into coordinates happen once per thread, later coordinates step from it.
template <int SPACE, class Dims, class Body>
__device__ __forceinline__ void batchForEach(const BatchScene* scenes, const BatchPlan* plan, Dims dims, Body body) {
    constexpr int K = batchPerThread(SPACE);
    const int n = plan->scenes;
    const int s = batchSceneOf(plan->start[SPACE], n);
    const BatchScene& B = scenes[s];
    const int count = B.count[SPACE];
    const int first = (static_cast<int>(blockIdx.x) - __ldg(plan->start[SPACE] + s)) * kBatchThreads * K + static_cast<int>(threadIdx.x);
    if (first >= count) return;
    int w, h;
    dims(B, w, h);
    const int row = first / w;
    int x = first - row * w, y = row % h, z = row / h;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = first + k * kBatchThreads;
        if (i >= count) break;
        body(B, i, x, y, z);
        x += kBatchThreads;
        while (x >= w) {
            x -= w;
            if (++y == h) {
                y = 0;
                ++z;
            }
        }
    }
}

__device__ __forceinline__ void cellDims(const BatchScene& B, int& w, int& h) {
    w = B.c.nx;
    h = B.c.ny;
}
__device__ __forceinline__ void faceDims(const BatchScene& B, int& w, int& h) {
    w = B.c.nx + 1;
    h = B.c.ny + 1;
}

__device__ __forceinline__ Velocity velocityOf(FaceT* const (&f)[3]) { return Velocity{f[0], f[1], f[2]}; }

}  // namespace

__global__ void __launch_bounds__(kBatchThreads) batchAdvectVelocity(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchFaces>(scenes, plan, faceDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgAdvectVelocityAt(B.adv[0], B.adv[1], B.adv[2], B.vel, B.c, x, y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchAdvectScalars(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchCells>(scenes, plan, cellDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgAdvectScalarsAt(B.aOut, B.aIn, velocityOf(B.adv), B.c, x, y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchVorticity(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchCells>(scenes, plan, cellDims, [](const BatchScene& B, int, int x, int y, int z) {
        if (B.c.eps == 0.0f) return;
        cfgVorticityAt(B.vort, velocityOf(B.adv), B.c, x, y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchCellForce(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchCells>(scenes, plan, cellDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgCellForceAt(B.force, B.vort, B.aOut, B.noise, B.c, x, y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchApplyForces(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchFaces>(scenes, plan, faceDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgApplyForcesAt(B.forced[0], B.forced[1], B.forced[2], velocityOf(B.adv), B.force, B.c, x, y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchPrepareIncrement(const BatchScene* __restrict__ scenes,
                                                                      const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchCells>(scenes, plan, cellDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgPrepareIncrementAt(B.proj[0], B.proj[1], B.proj[2], velocityOf(B.forced), B.pressure, B.divergence, B.c.nx, B.c.ny, B.c.nz, x,
                              y, z);
    });
}

__global__ void __launch_bounds__(kBatchThreads) batchSubtractIncrement(const BatchScene* __restrict__ scenes,
                                                                       const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchCells>(scenes, plan, cellDims, [](const BatchScene& B, int, int x, int y, int z) {
        cfgSubtractIncrementAt(B.proj[0], B.proj[1], B.proj[2], B.delta, B.c.nx, B.c.ny, B.c.nz, 1, x, y, z);
    });
}

// Warps of 32 consecutive elements are whole: a scene's count is a multiple of 32.
__global__ void __launch_bounds__(kBatchThreads) batchOccupancy(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchBricks>(
        scenes, plan,
        [](const BatchScene&, int& w, int& h) {
            w = 32;
            h = 1 << 30;
        },
        [](const BatchScene& B, int, int lane, int unit, int) { cfgOccupancyAt(B.occupancy, B.aOut, nullptr, B.c, unit, 1 << 30, lane); });
}

__global__ void __launch_bounds__(kBatchThreads) batchTransmittance(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchLight>(
        scenes, plan,
        [](const BatchScene& B, int& w, int& h) {
            w = B.c.lx;
            h = B.c.ly;
        },
        [](const BatchScene& B, int, int x, int y, int z) { cfgTransmittanceAt<1, true>(B.transmittance, B.aOut, B.occupancy, B.c, x, y, z, 0, true); });
}

__global__ void __launch_bounds__(kBatchThreads) batchRaymarch(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchPixels>(
        scenes, plan,
        [](const BatchScene& B, int& w, int& h) {
            w = B.c.frameW;
            h = B.c.frameH;
        },
        [](const BatchScene& B, int, int x, int y, int) { cfgRaymarchAt<1, true>(B.hdr, B.aOut, B.transmittance, B.occupancy, B.c, x, y, 0, true); });
}

__global__ void __launch_bounds__(kBatchThreads) batchPackHdr(const BatchScene* __restrict__ scenes, const BatchPlan* __restrict__ plan) {
    batchForEach<kBatchPixels>(
        scenes, plan,
        [](const BatchScene& B, int& w, int& h) {
            w = B.c.frameW;
            h = B.c.frameH;
        },
        [](const BatchScene& B, int i, int x, int y, int) {
            if (B.slot == nullptr) return;
            packHdrPixel(B.slot, B.slotPitch, B.slotFormat, B.hdr[i], x, y);
        });
}

}  // namespace firesim
