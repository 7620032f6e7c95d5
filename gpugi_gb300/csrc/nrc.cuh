// Neural radiance cache: a small MLP evaluated and trained on the tensor
// cores. No counterpart in the reference (a project addition).
//
// Network: 64 inputs -> 4 hidden layers of 64 (ReLU) -> 3 outputs (padded to
// 16), no biases (one input is a constant 1). FP16 weights and activations,
// FP32 accumulation. Inputs (64):
//   [0, 36)   position in the scene box, 6 octaves of sin/cos(2^k pi x) per axis
//   [36, 52)  outgoing direction, real spherical harmonics of degree < 4 (16)
//   [52, 55)  shading normal
//   [55, 58)  albedo
//   58        constant 1 (acts as the first layer's bias)
//   [59, 64)  zero padding
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace gpugi {
namespace nrc {

constexpr float kPI_F = 3.14159265358979f;
constexpr int kIn = 64, kHidden = 64, kOutPad = 16, kLayers = 5;
// Weight matrix l maps kIn (64) -> kHidden (64) for l < 4 and 64 -> 16 for l = 4.
GPUGI_HD constexpr int out_of(int l) { return l == 4 ? 16 : 64; }
constexpr int kParams = 4 * 64 * 64 + 64 * 16;  // 17,408
// Offset of layer l in a flat parameter array (row-major [in][out]).
GPUGI_HD constexpr int layer_offset(int l) { return l * 64 * 64; }
// Shared-memory row stride (in halves) of the staged weights: 72 = 64 + 8
// keeps the 8 fragment rows of a warp on different banks.
constexpr int kRow = 72;

struct Query {  // one cache lookup / training sample
    float3 pos, dir, normal, albedo;
};

// Frequency + spherical-harmonics encoding of one query, in 16-byte chunks of
// eight features (chunk c = features [8 c, 8 c + 8)), so that threads can share a
// query and store it chunk by chunk.
struct EncodeInput {
    float f[3];    // pi x position in the box; octave o of an axis is f 2^o, exactly
    float sh[16];
    float rest[7];
};
GPUGI_D EncodeInput encode_input(const Query& q, float3 boxMin, float3 boxInvExtent) {
    EncodeInput e;
    const float p[3] = {(q.pos.x - boxMin.x) * boxInvExtent.x, (q.pos.y - boxMin.y) * boxInvExtent.y,
                        (q.pos.z - boxMin.z) * boxInvExtent.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) e.f[d] = kPI_F * p[d];
    const float x = q.dir.x, y = q.dir.y, z = q.dir.z;
    const float xx = x * x, yy = y * y, zz = z * z;
    const float sh[16] = {0.28209479f,
                          -0.48860251f * y, 0.48860251f * z, -0.48860251f * x,
                          1.09254843f * x * y, -1.09254843f * y * z, 0.31539157f * (3.0f * zz - 1.0f),
                          -1.09254843f * x * z, 0.54627422f * (xx - yy),
                          0.59004359f * y * (-3.0f * xx + yy), 2.89061144f * x * y * z,
                          0.45704580f * y * (1.0f - 5.0f * zz), 0.37317633f * z * (5.0f * zz - 3.0f),
                          0.45704580f * x * (1.0f - 5.0f * zz), 1.44530572f * z * (xx - yy),
                          0.59004359f * x * (-xx + 3.0f * yy)};
#pragma unroll
    for (int i = 0; i < 16; ++i) e.sh[i] = sh[i];
    const float rest[7] = {q.normal.x, q.normal.y, q.normal.z, q.albedo.x, q.albedo.y, q.albedo.z, 1.0f};
#pragma unroll
    for (int i = 0; i < 7; ++i) e.rest[i] = rest[i];
    return e;
}
template <int C>
GPUGI_D uint4 encode_chunk(const EncodeInput& e) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = 8 * C + 2 * i;  // features k, k + 1
        float a, b;
        if (k < 36) {
            sincosf(e.f[k / 12] * (float)(1 << (k % 12 / 2)), &a, &b);
        } else {
            auto get = [&](int j) { return j < 52 ? e.sh[j < 52 ? j - 36 : 0] : j < 59 ? e.rest[j >= 52 && j < 59 ? j - 52 : 0] : 0.0f; };
            a = get(k);
            b = get(k + 1);
        }
        __half2 h = __floats2half2_rn(a, b);
        w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// All chunks of a query; out is 16-byte aligned.
GPUGI_D void encode(const Query& q, float3 boxMin, float3 boxInvExtent, __half* out) {
    const EncodeInput e = encode_input(q, boxMin, boxInvExtent);
    uint4* o = reinterpret_cast<uint4*>(out);
    o[0] = encode_chunk<0>(e);
    o[1] = encode_chunk<1>(e);
    o[2] = encode_chunk<2>(e);
    o[3] = encode_chunk<3>(e);
    o[4] = encode_chunk<4>(e);
    o[5] = encode_chunk<5>(e);
    o[6] = encode_chunk<6>(e);
    o[7] = encode_chunk<7>(e);
}

}  // namespace nrc
}  // namespace gpugi
