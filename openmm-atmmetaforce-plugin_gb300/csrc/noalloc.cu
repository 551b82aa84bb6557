// Reaction-field nonbonded energy and forces for callers that cannot allocate
// device memory.
//
// Some callers of this library run where cudaMalloc is not an option: code
// that owns all device memory through its own pool or arena, code running
// while another component forbids new allocations (a memory budget already
// handed out, an allocator that must not be re-entered), or host code that
// simply must not add allocation latency to its step.  They get this one entry
// point, which takes every input and output from the caller and keeps its
// scratch (64-bit fixed-point force accumulators, FP32 positions and parameters,
// block boxes and per-CTA energy partials) in a file-scope __device__ array that every GPU loading the library holds
// until the process exits.
//
// It is the all-pairs variant of the pair-tile kernel of kernels.cu for
// CutoffPeriodic (reaction field) with exclusions, for at most
// kNoAllocMaxAtoms particles.  The rest of the library is untouched by it.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>
#include <string>

#include "../../include/atm_capi.h"
#include "model.h"

namespace atm {
namespace {

constexpr int kNoAllocMaxAtoms = 16384;  // particles per call
constexpr int kNoAllocCtas = 512;        // CTAs of the tile pass (one energy partial each)
constexpr int kNoAllocThreads = 256;
constexpr int kMaxDevices = 64;
constexpr double kFix = 4294967296.0;  // 2^32 fixed-point units per kJ/mol/nm

struct NoAllocScratch {
    unsigned long long force[3 * kNoAllocMaxAtoms];
    float4 posq[kNoAllocMaxAtoms];      // position in the cell, charge * sqrt(k_e)
    float2 lj[kNoAllocMaxAtoms];        // sigma / 2, 2 sqrt(epsilon)
    float4 box_c[kNoAllocMaxAtoms / 32];  // bounding boxes of the blocks of 32 particles: centres
    float4 box_h[kNoAllocMaxAtoms / 32];  //   and half extents
    double energy[kNoAllocCtas];
};

// The scratch every call shares (about 800 KB per GPU).
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

std::mutex g_setup_mutex;
NoAllocScratch* g_scratch_ptr[kMaxDevices] = {nullptr};

// Per particle, once: the FP32 position in the cell and parameters that every tile
// reads, and zeroed forces; per block of 32 (a warp): the bounding box around its
// first particle's periodic image.
__global__ void __launch_bounds__(kNoAllocThreads) k_noalloc_prepare(
    NoAllocScratch* s, int n, const double* __restrict__ pos, const double* __restrict__ q,
    const double* __restrict__ sig, const double* __restrict__ eps, double Lx, double Ly, double Lz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if (i - lane >= n) return;
    const bool vi = i < n;
    float x = 0.f, y = 0.f, z = 0.f;
    if (vi) {
        const float sqk = 11.787089759563214f;  // sqrt(138.935456)
        x = (float)(pos[3 * i] - Lx * floor(pos[3 * i] / Lx));
        y = (float)(pos[3 * i + 1] - Ly * floor(pos[3 * i + 1] / Ly));
        z = (float)(pos[3 * i + 2] - Lz * floor(pos[3 * i + 2] / Lz));
        s->posq[i] = make_float4(x, y, z, (float)q[i] * sqk);
        s->lj[i] = make_float2(0.5f * (float)sig[i], 2.0f * sqrtf((float)eps[i]));
        for (int a = 0; a < 3; a++) s->force[a * n + i] = 0ull;
    }
    const float fL[3] = {(float)Lx, (float)Ly, (float)Lz};
    float r[3] = {x, y, z}, c[3], h[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float r0 = __shfl_sync(0xffffffffu, r[a], 0);
        float d = vi ? r[a] - r0 : 0.f;
        d -= fL[a] * rintf(d / fL[a]);
        float lo = d, hi = d;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        c[a] = r0 + 0.5f * (lo + hi);
        h[a] = 0.5f * (hi - lo);
    }
    if (lane == 0) {
        s->box_c[i >> 5] = make_float4(c[0], c[1], c[2], 0.f);
        s->box_h[i >> 5] = make_float4(h[0], h[1], h[2], 0.f);
    }
}

__device__ __forceinline__ void tri_index(long long t, int nb, int& I, int& J) {
    // tile t of the upper triangle (I <= J) of an nb x nb block grid, row-major
    long long lo = 0, hi = nb - 1;
    while (lo < hi) {  // largest I with first(I) <= t, first(I) = I*nb - I*(I-1)/2
        long long mid = (lo + hi + 1) >> 1;
        long long first = mid * nb - mid * (mid - 1) / 2;
        if (first <= t) lo = mid;
        else hi = mid - 1;
    }
    I = (int)lo;
    long long first = lo * nb - lo * (lo - 1) / 2;
    J = (int)(lo + (t - first));
}

// Smallest distance along one axis between two boxes on a periodic axis (never
// more than the true one: rounding is covered by the slack).
__device__ __forceinline__ float axis_gap(float ci, float cj, float h, float L, float iL, float slack) {
    float d = cj - ci;
    d -= L * rintf(d * iL);
    return fmaxf(0.f, fabsf(d) - h - slack);
}

// Each lane of a warp tests one tile of the upper triangle (block I, block J) by its
// blocks' boxes, tiles gw, gw + nw, ... so that neighbouring tiles, which are alike,
// go to different warps; the tiles within the cutoff are then evaluated one by one,
// 32 x 32 pairs: a first loop marks the pairs within the cutoff (bit k of lane l: the
// pair of i = l and j = (l + k) & 31), a second evaluates the steps k with any pair.
// A tile or step left out holds no counted pair, so the FP32 sums are the same bits as
// all pairs'.  12,000 particles: 471 us with every tile evaluated, FP64 wrapping and the
// exclusion lists read per pair, 63 us so (and 24 -> 3.5 us for the finish, whose 512
// energy partials one thread summed).  The energy's order of operations (fmaf) is
// written out so that the sums stay the same bits.
__global__ void __launch_bounds__(kNoAllocThreads) k_noalloc_tiles(
    NoAllocScratch* s, int n, const int* __restrict__ ex_start, const int* __restrict__ ex_list, double Lx, double Ly,
    double Lz, float rc2, float krf, float crf) {
    __shared__ double red[kNoAllocThreads / 32];
    __shared__ float4 s_p[kNoAllocThreads / 32][64];
    __shared__ float2 s_l[kNoAllocThreads / 32][64];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int nb = (n + 31) / 32;
    const long long ntiles = (long long)nb * (nb + 1) / 2;
    const float fLx = (float)Lx, fLy = (float)Ly, fLz = (float)Lz;
    const float iLx = 1.0f / fLx, iLy = 1.0f / fLy, iLz = 1.0f / fLz;
    const float slack = 1e-4f + 1e-6f * fmaxf(fLx, fmaxf(fLy, fLz));
    float4* sp = s_p[warp];
    float2* sl = s_l[warp];
    double ewarp = 0.0;
    for (long long base = gw; base < ntiles; base += 32ll * nw) {
        const long long t = base + (long long)lane * nw;
        int tI = 0, tJ = 0;
        bool near = t < ntiles;
        if (near) {
            tri_index(t, nb, tI, tJ);
            const float4 ci = s->box_c[tI], hi = s->box_h[tI], cj = s->box_c[tJ], hj = s->box_h[tJ];
            const float gx = axis_gap(ci.x, cj.x, hi.x + hj.x, fLx, iLx, slack);
            const float gy = axis_gap(ci.y, cj.y, hi.y + hj.y, fLy, iLy, slack);
            const float gz = axis_gap(ci.z, cj.z, hi.z + hj.z, fLz, iLz, slack);
            near = !(gx * gx + gy * gy + gz * gz >= rc2);  // (a box that is not a number is kept)
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, near); todo; todo &= todo - 1) {
            const int from = __ffs(todo) - 1;
            const int I = __shfl_sync(0xffffffffu, tI, from), J = __shfl_sync(0xffffffffu, tJ, from);
            const int i = I * 32 + lane, j0 = J * 32 + lane;
            const bool vi = i < n, diag = I == J;
            float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), pj = pi;
            float2 li = make_float2(0.f, 0.f), lj = li;
            unsigned excl = 0u;  // bit j - 32 J: excluded with i
            if (vi) {
                pi = s->posq[i];
                li = s->lj[i];
                for (int m = ex_start[i]; m < ex_start[i + 1]; m++) {
                    const int j = ex_list[m];
                    if (j >> 5 == J) excl |= 1u << (j & 31);
                }
            }
            if (j0 < n) {
                pj = s->posq[j0];
                lj = s->lj[j0];
            }
            __syncwarp();
            sp[lane] = sp[lane + 32] = pj;
            sl[lane] = sl[lane + 32] = lj;
            __syncwarp();
            unsigned in = 0u;
#pragma unroll 8
            for (int k = 0; k < 32; k++) {
                const float4 p = sp[lane + k];
                float dx = p.x - pi.x, dy = p.y - pi.y, dz = p.z - pi.z;
                dx -= fLx * rintf(dx * iLx);
                dy -= fLy * rintf(dy * iLy);
                dz -= fLz * rintf(dz * iLz);
                const float r2 = dx * dx + dy * dy + dz * dz;
                in |= r2 < rc2 ? 1u << k : 0u;
            }
            // not counted: padding, the particle with itself, exclusions (their bit
            // j - 32 J taken to the lane's order, k = (j - l) & 31)
            const int nj = min(32, n - J * 32);
            const unsigned valid = nj >= 32 ? 0xffffffffu : (1u << nj) - 1u;
            const unsigned drop = excl | ~valid;
            in &= ~__funnelshift_r(drop, drop, lane);
            if (diag) in &= ~1u;
            if (!vi) in = 0u;
            unsigned steps = __reduce_or_sync(0xffffffffu, in);
            if (!steps) continue;
            float fix = 0.f, fiy = 0.f, fiz = 0.f, fjx = 0.f, fjy = 0.f, fjz = 0.f;
            double e = 0.0;
            int at = 0;  // the j force held by lane l is that of j = (l + at) & 31
            for (; steps; steps &= steps - 1) {
                const int k = __ffs(steps) - 1, src = (lane + k - at) & 31;
                fjx = __shfl_sync(0xffffffffu, fjx, src);
                fjy = __shfl_sync(0xffffffffu, fjy, src);
                fjz = __shfl_sync(0xffffffffu, fjz, src);
                at = k;
                if ((in >> k) & 1u) {
                    const float4 p = sp[lane + k];
                    const float2 l = sl[lane + k];
                    float dx = p.x - pi.x, dy = p.y - pi.y, dz = p.z - pi.z;
                    dx -= fLx * rintf(dx * iLx);
                    dy -= fLy * rintf(dy * iLy);
                    dz -= fLz * rintf(dz * iLz);
                    float r2 = dx * dx + dy * dy + dz * dz;
                    float invr = rsqrtf(r2), invr2 = invr * invr;
                    float sg = li.x + l.x;
                    float s2 = sg * sg * invr2, s6 = s2 * s2 * s2;
                    float ep = li.y * l.y;
                    float qq = pi.w * p.w;
                    const float en = fmaf(qq, fmaf(krf, r2, invr) - crf, ep * fmaf(s6, s6, -s6));
                    float fr = ep * (12.0f * s6 * s6 - 6.0f * s6) * invr2 + qq * (invr * invr2 - 2.0f * krf);
                    e += (double)en;
                    fix -= fr * dx;
                    fiy -= fr * dy;
                    fiz -= fr * dz;
                    fjx += fr * dx;
                    fjy += fr * dy;
                    fjz += fr * dz;
                }
            }
            // back to the lane's own j
            const int src = (lane - at) & 31;
            fjx = __shfl_sync(0xffffffffu, fjx, src);
            fjy = __shfl_sync(0xffffffffu, fjy, src);
            fjz = __shfl_sync(0xffffffffu, fjz, src);
            ewarp += diag ? 0.5 * e : e;
            if (vi) {
                atomicAdd(&s->force[i], (unsigned long long)__float2ll_rn(fix * 4294967296.0f));
                atomicAdd(&s->force[n + i], (unsigned long long)__float2ll_rn(fiy * 4294967296.0f));
                atomicAdd(&s->force[2 * n + i], (unsigned long long)__float2ll_rn(fiz * 4294967296.0f));
            }
            if (!diag && j0 < n) {
                atomicAdd(&s->force[j0], (unsigned long long)__float2ll_rn(fjx * 4294967296.0f));
                atomicAdd(&s->force[n + j0], (unsigned long long)__float2ll_rn(fjy * 4294967296.0f));
                atomicAdd(&s->force[2 * n + j0], (unsigned long long)__float2ll_rn(fjz * 4294967296.0f));
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) ewarp += __shfl_xor_sync(0xffffffffu, ewarp, o);
    if (lane == 0) red[warp] = ewarp;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < kNoAllocThreads / 32; w++) sum += red[w];
        s->energy[blockIdx.x] = sum;  // one slot per CTA: no order dependence
    }
}

__global__ void k_noalloc_finish(const NoAllocScratch* s, int n, double* energy, double* forces) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        for (int a = 0; a < 3; a++)
            forces[3 * k + a] = (double)(long long)s->force[a * n + k] * (1.0 / kFix);
    }
    // the CTAs' energies by the first warp, in a fixed order
    if (k < 32) {
        double sum = 0.0;
        for (int c = k; c < kNoAllocCtas; c += 32) sum += s->energy[c];
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (k == 0) *energy = sum;
    }
}

// Device address of the scratch on the current device, looked up once per
// device (cudaGetSymbolAddress with that device current).
NoAllocScratch* scratch_for_current_device() {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) throw Error(ATM_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(err));
    if (dev < 0 || dev >= kMaxDevices) throw Error(ATM_ERR_UNSUPPORTED, "device ordinal too large");
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (err != cudaSuccess)
            throw Error(ATM_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(err));
        g_scratch_ptr[dev] = (NoAllocScratch*)p;
    }
    return g_scratch_ptr[dev];
}

}  // namespace

// Records the message returned by atm_last_error() (defined with the other entry points).
void set_last_error(const std::string& msg);

}  // namespace atm

extern "C" int atm_rf_nonbonded_noalloc(int n, const double* d_pos, const double* d_charge, const double* d_sigma,
                                        const double* d_epsilon, const int* d_excl_start, const int* d_excl,
                                        const double* box, double cutoff, double eps_rf, double* d_energy,
                                        double* d_forces, void* stream) {
    using namespace atm;
    try {
        if (n <= 0 || !d_pos || !d_charge || !d_sigma || !d_epsilon || !d_excl_start || !d_excl || !box ||
            !d_energy || !d_forces)
            throw Error(ATM_ERR_INVALID_ARGUMENT, "null pointer or empty system");
        if (n > kNoAllocMaxAtoms)
            throw Error(ATM_ERR_INVALID_ARGUMENT,
                        "atm_rf_nonbonded_noalloc: " + std::to_string(n) + " particles exceed the maximum of " +
                            std::to_string(kNoAllocMaxAtoms));
        if (!(cutoff > 0) || !(eps_rf > 0)) throw Error(ATM_ERR_INVALID_ARGUMENT, "bad cutoff or dielectric");
        for (int a = 0; a < 3; a++)
            if (!(box[a] >= 2.0 * cutoff))
                throw Error(ATM_ERR_INVALID_ARGUMENT, "the box must be at least twice the cutoff");
        NoAllocScratch* s = scratch_for_current_device();
        cudaStream_t st = (cudaStream_t)stream;
        double krf = (eps_rf - 1.0) / ((2.0 * eps_rf + 1.0) * cutoff * cutoff * cutoff);
        double crf = 3.0 * eps_rf / ((2.0 * eps_rf + 1.0) * cutoff);
        const int blocks = (n + kNoAllocThreads - 1) / kNoAllocThreads;
        k_noalloc_prepare<<<blocks, kNoAllocThreads, 0, st>>>(s, n, d_pos, d_charge, d_sigma, d_epsilon, box[0], box[1],
                                                              box[2]);
        k_noalloc_tiles<<<kNoAllocCtas, kNoAllocThreads, 0, st>>>(s, n, d_excl_start, d_excl, box[0], box[1], box[2],
                                                                  (float)(cutoff * cutoff), (float)krf, (float)crf);
        k_noalloc_finish<<<blocks, kNoAllocThreads, 0, st>>>(s, n, d_energy, d_forces);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) throw Error(ATM_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(err));
        set_last_error("");
        return ATM_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    }
}
