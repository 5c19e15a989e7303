// The reference's element of a crystal that stands alone (PESysMatGen.cu:1207-1231, :1329-1359: self
// attenuation, absorption, solid angle; unrotated) behind a plate without holes or attenuation (:1240-1254: a
// ray whose chord in it is below 0.1 mm does not count), one rounding at a time, one thread per voxel.
// Arguments: crystal x y z (y with the FOV offset), width thickness height, mu, mu_pe, the plate's box x1 y1 z1
// x2 y2 z2 (x1 > x2: none), then x y z of each voxel.
// Prints the bits of each element.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include <cuda_runtime.h>

#define ADD __fadd_rn
#define SUB __fsub_rn
#define MUL __fmul_rn
#define DIV __fdiv_rn
#define FMA __fmaf_rn

struct Crystal {
    float pos[3], size[3], mu, mu_pe, plate[6];
};

// centre, centre - voxel, lower and upper face - voxel of part i of n along an axis
__device__ void part(int i, float n, float size, float p, float* r)
{
    r[0] = ADD(-size / 2.0f, MUL(DIV((float)i + 0.5f, n), size));
    r[1] = SUB(r[0], p);
    r[2] = SUB(MUL(SUB(DIV((float)i, n), 0.5f), size), p);
    r[3] = SUB(MUL(SUB(DIV((float)i + 1.0f, n), 0.5f), size), p);
}

__device__ float norm(float x, float y, float z) { return FMA(z, z, FMA(y, y, MUL(x, x))); }

__device__ void clip(float lo, float hi, float inv, float& t0, float& t1)
{
    const float u = MUL(lo, inv), v = MUL(hi, inv);
    t0 = fmaxf(t0, fminf(u, v));
    t1 = fminf(t1, fmaxf(u, v));
}

__device__ float inside(float t0, float t1, float end)
{
    if (SUB(t1, t0) < 0.001f || t0 >= end || t1 <= 0.001f) return 0.0f;
    return SUB(fminf(t1, end), t0 > 0.001f ? t0 : 0.0f);
}

__global__ void elements(Crystal c, const float* voxel, int n, float* out)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    float p[3], total = 0.0f;
    for (int k = 0; k < 3; ++k) p[k] = SUB(voxel[3 * v + k], c.pos[k]);
    const float w = c.size[0], t = c.size[1], h = c.size[2];
    for (int s = 0; s < 1024; ++s) {
        float a[3][4];
        part((s >> 4) & 7, 8.0f, w, p[0], a[0]);
        part(s & 15, 16.0f, t, p[1], a[1]);
        part(s >> 7, 8.0f, h, p[2], a[2]);
        const float tio = __fsqrt_rn(norm(a[0][1], a[1][1], a[2][1]));
        float t0 = -INFINITY, t1 = INFINITY, u0 = -INFINITY, u1 = INFINITY, l0 = -INFINITY, l1 = INFINITY;
        float world[3], far[3], ext[3];
        for (int k = 0; k < 3; ++k) {
            const float inv = DIV(tio, a[k][1]);
            clip(SUB(-c.size[k] / 2.0f, p[k]), SUB(c.size[k] / 2.0f, p[k]), inv, t0, t1);
            clip(a[k][2], a[k][3], inv, u0, u1);
            world[k] = SUB(ADD(c.pos[k], a[k][0]), voxel[3 * v + k]);
        }
        if (c.plate[0] <= c.plate[3]) {
            float d[3], q0 = -INFINITY, q1 = INFINITY;
            for (int k = 0; k < 3; ++k) d[k] = SUB(ADD(c.pos[k], a[k][0]), voxel[3 * v + k]);
            const float len = __fsqrt_rn(norm(d[0], d[1], d[2]));
            for (int k = 0; k < 3; ++k)
                clip(SUB(c.plate[k], voxel[3 * v + k]), SUB(c.plate[3 + k], voxel[3 * v + k]), DIV(len, d[k]), q0, q1);
            const bool none = SUB(q1, q0) < 0.001f || q0 >= len || q1 >= len || q0 <= 0.001f || q1 <= 0.001f;
            if (none || SUB(q1, q0) < 0.1f) continue;
        }
        const float self = SUB(inside(t0, t1, tio), inside(u0, u1, tio));
        const float dsq = norm(world[0], world[1], world[2]), sq = __fsqrt_rn(dsq);
        for (int k = 0; k < 3; ++k) {
            far[k] = ADD(a[k][0], DIV(MUL(1000.0f, a[k][1]), sq));
            ext[k] = SUB(far[k], p[k]);
        }
        const float end = __fsqrt_rn(norm(ext[1], ext[0], ext[2]));
        for (int k = 0; k < 3; ++k) clip(a[k][2], a[k][3], DIV(end, ext[k]), l0, l1);
        const bool out_of = SUB(l1, l0) < 0.001f || l0 >= end || l1 >= end || l0 <= 0.001f || l1 <= 0.001f;
        const float labs = out_of ? 0.0f : SUB(l1, l0);
        const double rq = __drcp_rn(__dmul_rn(__dmul_rn(4.0 * 3.14159265358979323846, (double)dsq), (double)sq));
        const float area[3] = {DIV(DIV(MUL(t, h), 8.0f), 16.0f), DIV(DIV(MUL(w, h), 8.0f), 8.0f),
                               DIV(DIV(MUL(w, t), 8.0f), 16.0f)};
        double most = 0.0;
        for (int k = 0; k < 3; ++k) most = fmax(most, __dmul_rn((double)area[k], (double)fabsf(world[k])));
        const float angle = (float)__dmul_rn(most, rq);
        const float absorbed = DIV(MUL(SUB(1.0f, expf(-MUL(labs, c.mu))), c.mu_pe), c.mu);
        total = ADD(total, MUL(MUL(expf(-MUL(self, c.mu)), angle), absorbed));
    }
    out[v] = total;
}

int main(int argc, char** argv)
{
    std::vector<float> a;
    for (int i = 1; i < argc; ++i) a.push_back((float)std::atof(argv[i]));
    const int n = ((int)a.size() - 14) / 3;
    if (n < 1) return 1;
    const Crystal c{{a[0], a[1], a[2]}, {a[3], a[4], a[5]}, a[6], a[7], {a[8], a[9], a[10], a[11], a[12], a[13]}};
    float *voxel, *out;
    cudaMalloc(&voxel, 3 * n * sizeof(float));
    cudaMalloc(&out, n * sizeof(float));
    cudaMemcpy(voxel, &a[14], 3 * n * sizeof(float), cudaMemcpyHostToDevice);
    elements<<<(n + 31) / 32, 32>>>(c, voxel, n, out);
    std::vector<uint32_t> bits(n);
    if (cudaMemcpy(bits.data(), out, n * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    for (uint32_t b : bits) std::printf("%u\n", b);
    return 0;
}
