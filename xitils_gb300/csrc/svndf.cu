// SVNDF of a displacement map on the GPU: the precomputation of the displacement
// prefiltering sandbox (downsampleDisplacementTexture,
// Sandbox/PrefilteringForRenderingDisplacementMappedSurfaces/Main.cpp:391-470) with
// the reference's EM fit of a 4-lobe vMF mixture (approximateBySEM,
// Include/Xitils/VonMisesFisherDistribution.h:68-160), one warp per low texel.
//
// The reference runs this on OpenMP threads with one sampler per thread, so the
// stream a texel's initial lobes come from depends on scheduling; here low texel t
// draws them from the PCG stream (t, 0, seed). Everything else follows the
// reference's arithmetic in its order, unfused (this unit is compiled with
// -fmad=false): the block's normals in row-major order, the mean height as a
// sequential sum, the E-step over samples (responsibilities without the lobe
// weights, as the reference computes them), the M-step sums per lobe in sample
// order (four lanes per lobe), the signed convergence difference. The EM stops on a threshold, so the
// fit is chaotic at the last ulp: exp, pow, asin, sin and cos are the correctly
// rounded ones of crmath.cuh, which round as the C library does for all but a
// small fraction of arguments.
#include <algorithm>

#include "xgb_kernels.h"
#include "materials.cuh"

namespace xgb {
namespace {

constexpr int kSvMaxRate = 16;
constexpr int kSvWarps = 4;
// A texel takes a block of kSvWarps warps from this rate on, and at any rate in a map of few
// texels, where the latency of a step decides; a warp otherwise. A noisy map fitted by a
// warp / a block per texel, ms per call: 1024 x 1024 at rate 3 4.36 / 5.76, 5 3.63 / 4.06, 8 3.24 / 3.27,
// 10 4.62 / 3.57, 13 6.00 / 3.65; 300 x 300 at rate 3 (10,000 texels) 0.42 / 0.39, 5 0.58 / 0.38, 8
// 0.59 / 0.42, 13 1.05 / 0.55. The same bits: the sums keep their order.
constexpr int kSvTeamRate = 9;
constexpr int kSvTeamTexels = 10000;
constexpr int kSvStepMax = 100000;    // StepMax
constexpr float kSvKappaLimit = 1000;  // KappaLimit
constexpr float kSvDiffThreshold = 1e-6f;

// A texel's shared memory: the block's normals, then per sample and lobe the responsibility
// and its products with the normal (the terms of the M-step's sums), sized for the rate.
struct SvLobes {
    float mu[kSvndfLobes][3], kappa[kSvndfLobes], alpha[kSvndfLobes];
    float norm[kSvndfLobes];  // vMF normaliser of kappa
    float lastMu[kSvndfLobes][3], lastKappa[kSvndfLobes];
};
__host__ __device__ constexpr size_t svWarpBytes(int samples) {
    return (sizeof(SvLobes) + 15) / 16 * 16 + (size_t)samples * 16 + (size_t)samples * kSvndfLobes * 16;
}

// vMF() (VonMisesFisherDistribution.h:205-211), the factor that depends on kappa alone.
__device__ __forceinline__ float vmfNorm(float kappa) {
    if (kappa == 0.0f) return 1.0f / (4 * kPi);
    return kappa / (2 * kPi * (1.0f - crExpf(-2 * kappa)));
}
__device__ __forceinline__ float vmfLobe(V3 mu, float kappa, float norm, V3 omega) {
    if (kappa == 0.0f) return norm;
    return norm * crExpf(kappa * (dot(omega, mu) - 1.0f));
}

// The fit is bound by the latency of a step: a texel takes from tens to thousands of them
// one after the other, so the slowest texels decide. The sums of the M-step have to be
// taken in sample order; four lanes per lobe take one each (the responsibility and the
// three components), their terms already multiplied out by the E-step's lanes, instead of
// one lane per lobe taking all four; the normalisers are computed once per step instead
// of once per sample. A noisy 1024 x 1024 map at rate 8: 36.9 ms with FP64 exponentials,
// 4.9 with float pairs (crmath.cuh), 3.0 so (the whole call).
template <int WARPS>
__global__ void __launch_bounds__(32 * kSvWarps) k_svndfFit(TextureDev src, float scale, int rate, uint32_t seed,
                                                             int resU, int resV, float4* lobes, float4* low) {
    extern __shared__ __align__(16) unsigned char svRaw[];
    constexpr int kLanesPerTexel = 32 * WARPS;
    const int team = threadIdx.x / kLanesPerTexel, lane = threadIdx.x % kLanesPerTexel;
    const int t = blockIdx.x * (kSvWarps / WARPS) + team;
    auto sync = [] {
        if (WARPS == 1) __syncwarp();
        else __syncthreads();
    };
    if (t >= resU * resV) return;  // all lanes of the texel leave
    unsigned char* mine = svRaw + team * svWarpBytes(rate * rate);
    SvLobes& S = *reinterpret_cast<SvLobes*>(mine);
    float4* normal = reinterpret_cast<float4*>(mine + (sizeof(SvLobes) + 15) / 16 * 16);  // w: height
    float4* term = normal + rate * rate;
    const int px = t % resU, py = t / resU;
    const int x0 = px * rate, y0 = py * rate;
    const int wc = min(rate, src.w - x0), hc = min(rate, src.h - y0);
    const int n = wc * hc;
    // the block's normals (Main.cpp:418-431), row-major over the texels inside the map
    for (int k = lane; k < n; k += kLanesPerTexel) {
        const int x = x0 + k % wc, y = y0 + k / wc;
        const float su = texDiffUAt(src, x, y), sv = texDiffVAt(src, x, y);
        const V3 nn = normalize(V3(-su * scale, -sv * scale, 1.0f));
        normal[k] = make_float4(nn.x, nn.y, nn.z, texAt(src, x, y).x);
    }
    sync();
    if (lane == 0) {
        float r = 0.0f;
        for (int k = 0; k < n; ++k) r += normal[k].w;
        low[t] = make_float4(r / (float)n, 0.0f, 0.0f, 0.0f);
    }
    float4* out = lobes + (size_t)t * 5;
    if (n == 1) {  // VonMisesFisherDistribution.h:79-86
        if (lane < kSvndfLobes) out[lane] = make_float4(normal[0].x, normal[0].y, normal[0].z, kSvKappaLimit);
        if (lane == 0) out[4] = make_float4(1.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    if (lane == 0) {  // initial lobes (:89-98)
        Pcg rng;
        rng.seed((uint32_t)t, 0u, seed);
        for (int j = 0; j < kSvndfLobes; ++j) {
            const float u = rng.randf();
            const float v = rng.randf();
            const float theta = crAsinf(u);
            const float phi = crMinusPi(2.0f * kPi * v);
            float st, ct, sp, cp;
            crSinCosf(theta, &st, &ct);
            crSinCosf(phi, &sp, &cp);
            S.mu[j][0] = ct * cp;
            S.mu[j][1] = ct * sp;
            S.mu[j][2] = st;
            S.kappa[j] = 0.5f;
            S.norm[j] = vmfNorm(0.5f);
            S.alpha[j] = 1.0f / kSvndfLobes;
        }
    }
    sync();
    for (int step = 0; step < kSvStepMax; ++step) {
        // E-step (:106-119)
        if (WARPS > 1) {
            // a lane per sample and lobe; the four lobes of a sample are neighbours
            const int l = lane & 3;
            const V3 mu(S.mu[l][0], S.mu[l][1], S.mu[l][2]);
            const float kappa = S.kappa[l], norm = S.norm[l];
            for (int base = 0; base < kSvndfLobes * n; base += kLanesPerTexel) {
                const int item = base + lane, i = min(item >> 2, n - 1);
                const float4 s4 = normal[i];
                const float v = vmfLobe(mu, kappa, norm, V3(s4.x, s4.y, s4.z));
                float gamma = 0.0f;
#pragma unroll
                for (int j = 0; j < kSvndfLobes; ++j) gamma += __shfl_sync(0xFFFFFFFFu, v, (lane & 28) + j);
                const float z = gamma > 0.0f ? v / gamma : 0.0f;
                if (item < kSvndfLobes * n) term[item] = make_float4(z, z * s4.x, z * s4.y, z * s4.z);
            }
        } else {
            V3 mu[kSvndfLobes];
            float kappa[kSvndfLobes], norm[kSvndfLobes];
#pragma unroll
            for (int j = 0; j < kSvndfLobes; ++j) {
                mu[j] = V3(S.mu[j][0], S.mu[j][1], S.mu[j][2]);
                kappa[j] = S.kappa[j];
                norm[j] = S.norm[j];
            }
            for (int i = lane; i < n; i += 32) {
                const float4 s4 = normal[i];
                const V3 s(s4.x, s4.y, s4.z);
                float v[kSvndfLobes];
                float gamma = 0.0f;
#pragma unroll
                for (int j = 0; j < kSvndfLobes; ++j) {
                    v[j] = vmfLobe(mu[j], kappa[j], norm[j], s);
                    gamma += v[j];
                }
#pragma unroll
                for (int j = 0; j < kSvndfLobes; ++j) {
                    const float z = gamma > 0.0f ? v[j] / gamma : 0.0f;
                    term[i * kSvndfLobes + j] = make_float4(z, z * s.x, z * s.y, z * s.z);
                }
            }
        }
        sync();
        // M-step (:121-138): lane 4 j + c sums term c of lobe j in sample order
        if (lane < 32) {
            const int j = (lane >> 2) & 3, c = lane & 3;
            float sum = 0.0f;
            {
                const float* p = reinterpret_cast<const float*>(term) + 4 * j + c;
                int i = 0;
                for (; i + 8 <= n; i += 8) {
                    float x[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[k] = p[16 * (i + k)];
#pragma unroll
                    for (int k = 0; k < 8; ++k) sum += x[k];
                }
                for (; i < n; ++i) sum += p[16 * i];
            }
            const int first = lane & ~3;
            const float a = __shfl_sync(0xFFFFFFFFu, sum, first);
            V3 r(__shfl_sync(0xFFFFFFFFu, sum, first + 1), __shfl_sync(0xFFFFFFFFu, sum, first + 2),
                 __shfl_sync(0xFFFFFFFFu, sum, first + 3));
            r = r / a;
            const float len = length(r);
            float k = (3 * len - crCubef(len)) / (1.0f - dot(r, r));
            const V3 m = normalize(r);
            if (k > kSvKappaLimit) k = kSvKappaLimit;
            if (k < 0.0f) k = 0.0f;
            const float nk = vmfNorm(k);
            if (lane < 4 * kSvndfLobes) {
                if (c == 0) {
                    S.kappa[j] = k;
                    S.norm[j] = nk;
                    S.alpha[j] = a / (float)n;
                } else {
                    S.mu[j][c - 1] = c == 1 ? m.x : c == 2 ? m.y : m.z;
                }
            }
        }
        sync();
        // convergence (:140-147): a signed sum, as in the reference; every lane the same
        bool done = false;
        if (step > 0) {
            float diff = 0.0f;
#pragma unroll
            for (int l = 0; l < kSvndfLobes; ++l) {
                const V3 d(S.mu[l][0] - S.lastMu[l][0], S.mu[l][1] - S.lastMu[l][1], S.mu[l][2] - S.lastMu[l][2]);
                diff += dot(d, d);
                diff += (S.kappa[l] - S.lastKappa[l]) * 0.1f;
            }
            done = diff < kSvDiffThreshold;
        }
        if (done) break;
        sync();
        if (lane < kSvndfLobes) {
            S.lastMu[lane][0] = S.mu[lane][0]; S.lastMu[lane][1] = S.mu[lane][1]; S.lastMu[lane][2] = S.mu[lane][2];
            S.lastKappa[lane] = S.kappa[lane];
        }
    }
    sync();
    if (lane < kSvndfLobes) out[lane] = make_float4(S.mu[lane][0], S.mu[lane][1], S.mu[lane][2], S.kappa[lane]);
    if (lane == 0) out[4] = make_float4(S.alpha[0], S.alpha[1], S.alpha[2], S.alpha[3]);
}

}  // namespace

cudaError_t svndfFit(const TextureDev& src, float scale, int rate, uint32_t seed, int resU, int resV, float4* lobes,
                     float4* low, cudaStream_t s) {
    if (rate < 1 || rate > kSvMaxRate) return cudaErrorInvalidValue;
    const int texels = resU * resV;
    const auto fit = [&](auto* kernel, int perBlock) {
        const size_t most = perBlock * svWarpBytes(kSvMaxRate * kSvMaxRate);
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
        kernel<<<(texels + perBlock - 1) / perBlock, 32 * kSvWarps, perBlock * svWarpBytes(rate * rate), s>>>(
            src, scale, rate, seed, resU, resV, lobes, low);
        return cudaGetLastError();
    };
    return rate >= kSvTeamRate || texels <= kSvTeamTexels ? fit(k_svndfFit<kSvWarps>, 1) : fit(k_svndfFit<1>, kSvWarps);
}

}  // namespace xgb
