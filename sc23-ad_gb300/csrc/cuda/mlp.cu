// The learned fractional-bit selector: a 3-layer FP32 MLP (in -> H -> H -> out,
// ReLU after the two hidden layers) trained and evaluated by these kernels.
//
// The reference picks F_G by a fixed rule (Work/main.cpp:153-161) or by a
// manual sweep (Work/sub.cpp:36-102, Work/run_sub.sh); it has no learned part,
// so this file has no reference counterpart.  The network maps matrix features
// to one predicted cost per candidate F (log2 of the iteration count of the
// integer solver); the selector takes the argmin.
//
// Every kernel reduces in a fixed order (no atomics), so training is
// reproducible run to run.  Parameter layout (one flat float array):
//   W1[H][I] b1[H] W2[H][H] b2[H] W3[O][H] b3[O]
#include <cmath>
#include <cstring>
#include <vector>

#include "../sagb_internal.hpp"
#include "common.cuh"

namespace sagb {

constexpr int kTile = 16;

// Y[b][n] = act(sum_k X[b][k] W[n][k] + bias[n]), k summed in increasing order.
__global__ void k_dense_fwd(const float *__restrict__ X, const float *__restrict__ W,
                            const float *__restrict__ bias, float *__restrict__ Y, int B, int K, int N, int relu) {
    __shared__ float sx[kTile][kTile + 1], sw[kTile][kTile + 1];
    const int tb = threadIdx.y, tn = threadIdx.x;
    const int b = blockIdx.y * kTile + tb, n = blockIdx.x * kTile + tn;
    float acc = 0.f;
    for (int k0 = 0; k0 < K; k0 += kTile) {
        const int kx = k0 + tn;
        sx[tb][tn] = (b < B && kx < K) ? X[(size_t)b * K + kx] : 0.f;
        const int nw = blockIdx.x * kTile + tb;
        sw[tb][tn] = (nw < N && kx < K) ? W[(size_t)nw * K + kx] : 0.f;
        __syncthreads();
        const int kk = min(kTile, K - k0);
        for (int t = 0; t < kk; t++) acc = __fmaf_rn(sx[tb][t], sw[tn][t], acc);
        __syncthreads();
    }
    if (b < B && n < N) {
        float y = acc + bias[n];
        if (relu) y = fmaxf(y, 0.f);
        Y[(size_t)b * N + n] = y;
    }
}

// dX[b][k] = (sum_n dY[b][n] W[n][k]) * (A[b][k] > 0), n in increasing order.
// A is the layer's input activation (post-ReLU), so the product is the
// gradient with respect to the previous layer's pre-activation.
__global__ void k_dense_bwd_x(const float *__restrict__ dY, const float *__restrict__ W,
                              const float *__restrict__ A, float *__restrict__ dX, int B, int N, int K) {
    __shared__ float sd[kTile][kTile + 1], sw[kTile][kTile + 1];
    const int tb = threadIdx.y, tk = threadIdx.x;
    const int b = blockIdx.y * kTile + tb, k = blockIdx.x * kTile + tk;
    float acc = 0.f;
    for (int n0 = 0; n0 < N; n0 += kTile) {
        const int nd = n0 + tk;
        sd[tb][tk] = (b < B && nd < N) ? dY[(size_t)b * N + nd] : 0.f;
        const int nw = n0 + tb;
        sw[tb][tk] = (nw < N && k < K) ? W[(size_t)nw * K + k] : 0.f;
        __syncthreads();
        const int nn = min(kTile, N - n0);
        for (int t = 0; t < nn; t++) acc = __fmaf_rn(sd[tb][t], sw[t][tk], acc);
        __syncthreads();
    }
    if (b < B && k < K) dX[(size_t)b * K + k] = A[(size_t)b * K + k] > 0.f ? acc : 0.f;
}

// dW[n][k] = sum_b dY[b][n] X[b][k]; db[n] = sum_b dY[b][n]; b in increasing order.
__global__ void k_dense_bwd_w(const float *__restrict__ dY, const float *__restrict__ X, float *__restrict__ dW,
                              float *__restrict__ db, int B, int N, int K) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < N * K) {
        const int n = idx / K, k = idx - n * K;
        float acc = 0.f;
        for (int b = 0; b < B; b++) acc = __fmaf_rn(dY[(size_t)b * N + n], X[(size_t)b * K + k], acc);
        dW[idx] = acc;
    } else if (idx < N * K + N) {
        const int n = idx - N * K;
        float acc = 0.f;
        for (int b = 0; b < B; b++) acc += dY[(size_t)b * N + n];
        db[n] = acc;
    }
}

// Masked mean squared error over one batch (one block):
//   L = sum M (Y - T)^2 / sum M,  dY = 2 M (Y - T) / sum M.
__global__ void k_mse(const float *__restrict__ Y, const float *__restrict__ T, const float *__restrict__ M,
                      float *__restrict__ dY, int count, float *__restrict__ loss) {
    __shared__ float sh[32];
    __shared__ float s_tot;
    float m = 0.f;
    for (int i = threadIdx.x; i < count; i += blockDim.x) m += M[i];
    // fixed-order block sum: warp shuffles, then warp 0 over the warp sums
    auto bsum = [&](float v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
            s_tot = t;
        }
        __syncthreads();
        const float r = s_tot;
        __syncthreads();
        return r;
    };
    const float msum = bsum(m);
    const float inv = msum > 0.f ? 1.f / msum : 0.f;
    float e = 0.f;
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const float d = Y[i] - T[i];
        e += M[i] * d * d;
        dY[i] = 2.f * M[i] * d * inv;
    }
    const float esum = bsum(e);
    if (threadIdx.x == 0) *loss = esum * inv;
}

// Adam (Kingma & Ba 2015) with bias correction; t is the 1-based step count.  The
// multiply-adds are written out: left to the compiler, each kernel fuses either product
// of a moment, and the weights after some steps depend on which.
__device__ __forceinline__ float adam_step(float w, float gi, float &m1, float &m2, float lr, float beta1, float beta2,
                                           float eps, float bc1, float bc2) {
    m1 = __fmaf_rn(1.f - beta1, gi, __fmul_rn(beta1, m1));
    m2 = __fmaf_rn(__fmul_rn(1.f - beta2, gi), gi, __fmul_rn(beta2, m2));
    const float mh = m1 / bc1, vh = m2 / bc2;
    return w - lr * mh / (sqrtf(vh) + eps);
}
__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                       float *__restrict__ m2, int n, float lr, float beta1, float beta2, float eps, float bc1,
                       float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float a = m1[i], v = m2[i];
    w[i] = adam_step(w[i], g[i], a, v, lr, beta1, beta2, eps, bc1, bc2);
    m1[i] = a;
    m2[i] = v;
}

// Xn[b][k] = (X[src(b)][k] - mu[k]) / sd[k]; rows gathered through perm (or
// taken in order when perm is null), targets and masks gathered alike.
__global__ void k_gather_norm(const float *__restrict__ X, const float *__restrict__ T, const float *__restrict__ M,
                              const int *__restrict__ perm, int off, int B, int I, int O,
                              const float *__restrict__ mu, const float *__restrict__ sd, float *__restrict__ Xb,
                              float *__restrict__ Tb, float *__restrict__ Mb) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = idx / (I + O), r = idx - b * (I + O);
    if (b >= B) return;
    const int s = perm ? perm[off + b] : off + b;
    if (r < I) {
        Xb[(size_t)b * I + r] = (X[(size_t)s * I + r] - mu[r]) / sd[r];
    } else if (T) {
        const int o = r - I;
        Tb[(size_t)b * O + o] = T[(size_t)s * O + o];
        Mb[(size_t)b * O + o] = M[(size_t)s * O + o];
    }
}

// -------------------------------------------------- an epoch in one launch
//
// Training steps on nets and batches that fit the shared memory: one cluster of
// kEpochCtas CTAs runs all mini-batches of an epoch, with two cluster barriers a
// step.  What bounded a step of eleven small kernels was their launches and
// chains of loads from L2 (about 80 us a step at 20-64-64-22 with 64 rows; half
// of the kernel time in k_dense_bwd_w).  Here the parameters live in every CTA's shared
// memory (rows padded to an odd stride: read along either index without bank
// conflicts).  A CTA takes the batch's rows blockwise through the forward and
// backward passes, which need no other rows, and writes its rows' activations
// and gradients into all CTAs.  After the first barrier each thread sums the
// gradient of its own parameter over the batch, updates it (moments in
// registers) and writes it into all CTAs; the second barrier ends the step.
// Every sum runs in the order of the kernels above.  A step at 20-64-64-22 with 32
// / 64 / 100 rows: 11.5 / 13.8 / 17.6 us; 1,109 rows, batches of 64, two epochs:
// 3,020 -> 590 us with the copies of the data.
constexpr int kEpochCtas = 8, kEpochThreads = 1024;
constexpr int kEpochParams = kEpochCtas * kEpochThreads;  // a parameter a thread
constexpr int kTrainRows = 1 << 18;                       // rows of the epochs prepared at a time
constexpr size_t kEpochSmem = 227 * 1024 - 512;           // (the rest is static)

struct EpochNet {
    int I, H, O;
    // padded parameters, in floats
    __host__ __device__ static int pad(int k) { return k | 1; }
    __host__ __device__ int b1() const { return H * pad(I); }
    __host__ __device__ int w2() const { return b1() + H; }
    __host__ __device__ int b2() const { return w2() + H * pad(H); }
    __host__ __device__ int w3() const { return b2() + H; }
    __host__ __device__ int b3() const { return w3() + O * pad(H); }
    __host__ __device__ int acts() const { return b3() + O; }
    __host__ __device__ int row() const { return I + 4 * H + 2 * O; }  // X, A1, A2, d1, d2, Y, dY
    __host__ __device__ size_t bytes(int B) const { return sizeof(float) * ((size_t)acts() + (size_t)B * row()); }
    int params() const { return H * I + H + H * H + H + O * H + O; }
};

__global__ void __launch_bounds__(kEpochThreads, 1)
k_epoch(EpochNet N, const float *__restrict__ X, const float *__restrict__ T, const float *__restrict__ M,
        const int *__restrict__ perm, int n, int batch, const float *__restrict__ mu, const float *__restrict__ sd,
        float *__restrict__ p, float *__restrict__ m1, float *__restrict__ m2, float *__restrict__ loss,
        const float2 *__restrict__ bc, float lr, float beta1, float beta2, float eps) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float sh[32];
    __shared__ float s_tot;
    const int tid = threadIdx.x, I = N.I, H = N.H, O = N.O;
    const unsigned rank = cluster_rank();
    unsigned other[kEpochCtas];  // this CTA's shared memory as the others see it: addresses in theirs
#pragma unroll
    for (int r = 0; r < kEpochCtas; r++) other[r] = map_rank(smem_addr(sm), r);
    auto put = [&](int at, float v) {  // in every CTA
        sm[at] = v;
#pragma unroll
        for (int r = 0; r < kEpochCtas; r++)
            if (r != (int)rank)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(other[r] + 4u * at), "f"(v) : "memory");
    };
    // the parameter of this thread: flat index, place in shared memory, layer
    const int mine = (int)rank * kEpochThreads + tid;
    int at = -1, layer = 0, row = 0, col = -1;  // col < 0: a bias
    {
        int i = mine, base = 0;
        auto take = [&](int l, int out, int in) {
            if (at >= 0 || i < 0) return;
            const int st = EpochNet::pad(in);
            if (i < out * in) {
                layer = l;
                row = i / in;
                col = i - row * in;
                at = base + row * st + col;
            } else if (i < out * in + out) {
                layer = l;
                row = i - out * in;
                at = base + out * st + row;
            }
            i -= out * in + out;
            base += out * st + out;
        };
        take(1, H, I);
        take(2, H, H);
        take(3, O, H);
    }
    float w = 0.f, a1 = 0.f, a2 = 0.f;
    if (at >= 0) {
        w = p[mine];
        a1 = m1[mine];
        a2 = m2[mine];
    }
    cluster_sync_all();  // every CTA runs
    if (at >= 0) put(at, w);
    cluster_sync_all();

    // activations, whole batch
    const int oX = N.acts(), oA1 = oX + batch * I, oA2 = oA1 + batch * H, oD1 = oA2 + batch * H, oD2 = oD1 + batch * H,
              oY = oD2 + batch * H, oDY = oY + batch * O;
    auto bsum = [&](float v) {  // as in k_mse
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) sh[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            float t = 0.f;
            for (int q = 0; q < (kEpochThreads >> 5); q++) t += sh[q];
            s_tot = t;
        }
        __syncthreads();
        const float r = s_tot;
        __syncthreads();
        return r;
    };
    const int steps = (n + batch - 1) / batch;
    for (int s = 0; s < steps; s++) {
        const int off = s * batch, B = min(batch, n - off), R = (B + kEpochCtas - 1) / kEpochCtas;
        const int r0 = min(B, (int)rank * R), r1 = min(B, r0 + R), nr = r1 - r0;
        const int *src = perm + off;
        // rows of the batch, normalised
        for (int i = tid; i < nr * I; i += kEpochThreads) {
            const int b = r0 + i / I, k = i % I;
            put(oX + b * I + k, (X[(size_t)__ldg(src + b) * I + k] - mu[k]) / sd[k]);
        }
        float m = 0.f;
        for (int i = tid; i < B * O; i += kEpochThreads) m += M[(size_t)__ldg(src + i / O) * O + i % O];
        const float msum = bsum(m);
        const float inv = msum > 0.f ? 1.f / msum : 0.f;
        // two rows a thread
        auto forward = [&](int in, int K, int wt, int bias, int out, int width, bool relu, bool all) {
            const int st = EpochNet::pad(K), half = (nr + 1) / 2;
            for (int i = tid; i < half * width; i += kEpochThreads) {
                const int g = i / width, o = i - g * width, b0 = r0 + g, b1 = min(r1 - 1, b0 + half);
                const bool two = b0 + half < r1;
                const float *wr = sm + wt + o * st, *x0 = sm + in + b0 * K, *x1 = sm + in + b1 * K;
                float y0 = 0.f, y1 = 0.f;
#pragma unroll 8
                for (int k = 0; k < K; k++) {
                    y0 = __fmaf_rn(x0[k], wr[k], y0);
                    y1 = __fmaf_rn(x1[k], wr[k], y1);
                }
                y0 = y0 + sm[bias + o];
                y1 = y1 + sm[bias + o];
                if (relu) {
                    y0 = fmaxf(y0, 0.f);
                    y1 = fmaxf(y1, 0.f);
                }
                if (all) {
                    put(out + b0 * width + o, y0);
                    if (two) put(out + b1 * width + o, y1);
                } else {
                    sm[out + b0 * width + o] = y0;
                    if (two) sm[out + b1 * width + o] = y1;
                    if (rank != 0) {  // CTA 0 sums the loss
                        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(other[0] + 4u * (out + b0 * width + o)), "f"(y0)
                                     : "memory");
                        if (two)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(other[0] + 4u * (out + b1 * width + o)),
                                         "f"(y1)
                                         : "memory");
                    }
                }
            }
            __syncthreads();
        };
        forward(oX, I, 0, N.b1(), oA1, H, true, true);
        forward(oA1, H, N.w2(), N.b2(), oA2, H, true, true);
        forward(oA2, H, N.w3(), N.b3(), oY, O, false, false);
        for (int i = tid; i < nr * O; i += kEpochThreads) {
            const int b = r0 + i / O, o = i % O;
            const size_t g = (size_t)__ldg(src + b) * O + o;
            const float d = sm[oY + b * O + o] - T[g];
            put(oDY + b * O + o, 2.f * M[g] * d * inv);
        }
        __syncthreads();
        auto backward = [&](int dy, int width, int wt, int act, int out, int K) {
            const int st = EpochNet::pad(K), half = (nr + 1) / 2;
            for (int i = tid; i < half * K; i += kEpochThreads) {
                const int g = i / K, k = i - g * K, b0 = r0 + g, b1 = min(r1 - 1, b0 + half);
                const bool two = b0 + half < r1;
                const float *wc = sm + wt + k, *d0 = sm + dy + b0 * width, *d1 = sm + dy + b1 * width;
                float y0 = 0.f, y1 = 0.f;
#pragma unroll 8
                for (int o = 0; o < width; o++) {
                    y0 = __fmaf_rn(d0[o], wc[o * st], y0);
                    y1 = __fmaf_rn(d1[o], wc[o * st], y1);
                }
                put(out + b0 * K + k, sm[act + b0 * K + k] > 0.f ? y0 : 0.f);
                if (two) put(out + b1 * K + k, sm[act + b1 * K + k] > 0.f ? y1 : 0.f);
            }
            __syncthreads();
        };
        backward(oDY, O, N.w3(), oA2, oD2, H);
        backward(oD2, H, N.w2(), oA1, oD1, H);
        cluster_sync_all();
        // gradient and update of this thread's parameter
        if (at >= 0) {
            const int width = layer == 3 ? O : H, K = layer == 1 ? I : H;
            const float *d = sm + (layer == 1 ? oD1 : layer == 2 ? oD2 : oDY) + row;
            float g = 0.f;
            if (col >= 0) {
                const float *x = sm + (layer == 1 ? oX : layer == 2 ? oA1 : oA2) + col;
#pragma unroll 8
                for (int b = 0; b < B; b++) g = __fmaf_rn(d[b * width], x[b * K], g);
            } else {
#pragma unroll 8
                for (int b = 0; b < B; b++) g += d[b * width];
            }
            const float2 c = __ldg(bc + s);
            w = adam_step(w, g, a1, a2, lr, beta1, beta2, eps, c.x, c.y);
            put(at, w);
        }
        if (rank == 0) {
            float e = 0.f;
            for (int i = tid; i < B * O; i += kEpochThreads) {
                const size_t g = (size_t)__ldg(src + i / O) * O + i % O;
                const float d = sm[oY + i] - T[g];
                e += M[g] * d * d;
            }
            const float esum = bsum(e);
            if (tid == 0) loss[s] = esum * inv;
        }
        cluster_sync_all();
    }
    if (at >= 0) {
        p[mine] = w;
        m1[mine] = a1;
        m2[mine] = a2;
    }
}

// ------------------------------------------------------------------ host side

Mlp::Mlp(int in, int hidden, int out, uint64_t seed) : nin(in), hid(hidden), nout(out) {
    if (in < 1 || hidden < 1 || out < 1 || in > 4096 || hidden > 4096 || out > 4096)
        throw CudaError{"invalid MLP shape"};
    const size_t np = nparams();
    // He-uniform initialisation from a splitmix64 stream (identical on every host)
    std::vector<float> w(np, 0.f);
    uint64_t st = seed;
    auto next = [&]() {
        uint64_t z = (st += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](size_t off, int rows, int cols) {
        const double lim = std::sqrt(6.0 / cols);
        for (size_t i = 0; i < (size_t)rows * cols; i++) w[off + i] = (float)((2.0 * next() - 1.0) * lim);
    };
    fill(off_w1(), hid, nin);
    fill(off_w2(), hid, hid);
    fill(off_w3(), nout, hid);
    p = (float *)dmalloc(np * 4 * sizeof(float));
    g = p + np;
    m1 = g + np;
    m2 = m1 + np;
    SAGB_CUDA(cudaMemcpy(p, w.data(), np * sizeof(float), cudaMemcpyHostToDevice));
    SAGB_CUDA(cudaMemset(g, 0, 3 * np * sizeof(float)));
    std::vector<float> mu(nin, 0.f), sd(nin, 1.f);
    norm = (float *)dmalloc(2 * nin * sizeof(float));
    SAGB_CUDA(cudaMemcpy(norm, mu.data(), nin * sizeof(float), cudaMemcpyHostToDevice));
    SAGB_CUDA(cudaMemcpy(norm + nin, sd.data(), nin * sizeof(float), cudaMemcpyHostToDevice));
}

Mlp::~Mlp() {
    dfree(p);
    dfree(norm);
    dfree(ws);
    dfree(data);
    dfree(perm_d);
}

void Mlp::reserve(int B) {
    if (B <= ws_batch) return;
    dfree(ws);
    // Xb, A1, A2, Y, Tb, Mb, dY, d2, d1, loss
    const size_t n = (size_t)B * (nin + 4 * hid + 4 * nout) + 1;
    ws = (float *)dmalloc(n * sizeof(float));
    ws_batch = B;
}

void Mlp::forward_batch(Ctx &c, int B) {
    float *Xb = ws, *A1 = Xb + (size_t)ws_batch * nin, *A2 = A1 + (size_t)ws_batch * hid,
          *Y = A2 + (size_t)ws_batch * hid;
    const dim3 blk(kTile, kTile);
    auto grid = [&](int n) { return dim3((n + kTile - 1) / kTile, (B + kTile - 1) / kTile); };
    k_dense_fwd<<<grid(hid), blk, 0, c.stream>>>(Xb, p + off_w1(), p + off_b1(), A1, B, nin, hid, 1);
    k_dense_fwd<<<grid(hid), blk, 0, c.stream>>>(A1, p + off_w2(), p + off_b2(), A2, B, hid, hid, 1);
    k_dense_fwd<<<grid(nout), blk, 0, c.stream>>>(A2, p + off_w3(), p + off_b3(), Y, B, hid, nout, 0);
    c.launches += 3;
}

void Mlp::backward_batch(Ctx &c, int B) {
    float *Xb = ws, *A1 = Xb + (size_t)ws_batch * nin, *A2 = A1 + (size_t)ws_batch * hid,
          *Y = A2 + (size_t)ws_batch * hid, *Tb = Y + (size_t)ws_batch * nout, *Mb = Tb + (size_t)ws_batch * nout,
          *dY = Mb + (size_t)ws_batch * nout, *d2 = dY + (size_t)ws_batch * nout, *d1 = d2 + (size_t)ws_batch * hid,
          *loss = d1 + (size_t)ws_batch * hid;
    k_mse<<<1, 1024, 0, c.stream>>>(Y, Tb, Mb, dY, B * nout, loss);
    const dim3 blk(kTile, kTile);
    auto gridx = [&](int k) { return dim3((k + kTile - 1) / kTile, (B + kTile - 1) / kTile); };
    auto gw = [&](int n, int k) { return (n * k + n + 255) / 256; };
    k_dense_bwd_w<<<gw(nout, hid), 256, 0, c.stream>>>(dY, A2, g + off_w3(), g + off_b3(), B, nout, hid);
    k_dense_bwd_x<<<gridx(hid), blk, 0, c.stream>>>(dY, p + off_w3(), A2, d2, B, nout, hid);
    k_dense_bwd_w<<<gw(hid, hid), 256, 0, c.stream>>>(d2, A1, g + off_w2(), g + off_b2(), B, hid, hid);
    k_dense_bwd_x<<<gridx(hid), blk, 0, c.stream>>>(d2, p + off_w2(), A1, d1, B, hid, hid);
    k_dense_bwd_w<<<gw(hid, nin), 256, 0, c.stream>>>(d1, Xb, g + off_w1(), g + off_b1(), B, hid, nin);
    c.launches += 6;
}

float *Mlp::loss_slot() { return ws + (size_t)ws_batch * (nin + 4 * hid + 4 * nout); }

void Mlp::set_norm(const float *mu, const float *sd) {
    for (int i = 0; i < nin; i++)
        if (!(sd[i] > 0.f)) throw CudaError{"feature scale must be positive"};
    SAGB_CUDA(cudaMemcpy(norm, mu, nin * sizeof(float), cudaMemcpyHostToDevice));
    SAGB_CUDA(cudaMemcpy(norm + nin, sd, nin * sizeof(float), cudaMemcpyHostToDevice));
}

void Mlp::load(Ctx &c, const float *X, const float *T, const float *M, int n) {
    const size_t bytes = (size_t)n * (nin + 2 * nout) * sizeof(float);
    if (n > data_n) {
        dfree(data);
        data = (float *)dmalloc(bytes);
        data_n = n;
    }
    SAGB_CUDA(cudaMemcpyAsync(data, X, (size_t)n * nin * sizeof(float), cudaMemcpyDefault, c.stream));
    if (T) {
        SAGB_CUDA(cudaMemcpyAsync(data + (size_t)n * nin, T, (size_t)n * nout * sizeof(float), cudaMemcpyDefault,
                                  c.stream));
        SAGB_CUDA(cudaMemcpyAsync(data + (size_t)n * (nin + nout), M, (size_t)n * nout * sizeof(float),
                                  cudaMemcpyDefault, c.stream));
    }
    loaded_n = n;
}

void Mlp::gather(Ctx &c, const int *perm, int off, int B, bool targets) {
    const int n = loaded_n;
    const float *X = data, *T = targets ? data + (size_t)n * nin : nullptr,
                *M = targets ? data + (size_t)n * (nin + nout) : nullptr;
    float *Xb = ws, *Y = Xb + (size_t)ws_batch * (nin + 2 * hid), *Tb = Y + (size_t)ws_batch * nout,
          *Mb = Tb + (size_t)ws_batch * nout;
    const int tot = B * (nin + nout);
    k_gather_norm<<<(tot + 255) / 256, 256, 0, c.stream>>>(X, T, M, perm, off, B, nin, nout, norm, norm + nin, Xb,
                                                          Tb, Mb);
    c.launches++;
}

void Mlp::predict(Ctx &c, const float *X, int n, float *Y) {
    reserve(n);
    load(c, X, nullptr, nullptr, n);
    gather(c, nullptr, 0, n, false);
    forward_batch(c, n);
    const float *Yd = ws + (size_t)ws_batch * (nin + 2 * hid);
    SAGB_CUDA(cudaMemcpyAsync(Y, Yd, (size_t)n * nout * sizeof(float), cudaMemcpyDefault, c.stream));
    SAGB_CUDA(cudaStreamSynchronize(c.stream));
}

float Mlp::gradient(Ctx &c, const float *X, const float *T, const float *M, int n, float *grad) {
    reserve(n);
    load(c, X, T, M, n);
    gather(c, nullptr, 0, n, true);
    forward_batch(c, n);
    backward_batch(c, n);
    float loss = 0.f;
    SAGB_CUDA(cudaMemcpyAsync(&loss, loss_slot(), sizeof(float), cudaMemcpyDeviceToHost, c.stream));
    if (grad)
        SAGB_CUDA(cudaMemcpyAsync(grad, g, nparams() * sizeof(float), cudaMemcpyDefault, c.stream));
    SAGB_CUDA(cudaStreamSynchronize(c.stream));
    return loss;
}

void Mlp::launch_epoch(Ctx &c, const EpochNet &net, const int *perm, int n, int batch, float *loss, const float2 *bc,
                       float lr, float beta1, float beta2, float eps) {
    const size_t smem = net.bytes(batch);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kEpochCtas);
    cfg.blockDim = dim3(kEpochThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kEpochCtas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const float *x = data, *y = data + (size_t)loaded_n * nin, *m = data + (size_t)loaded_n * (nin + nout);
    SAGB_CUDA(cudaLaunchKernelEx(&cfg, k_epoch, net, x, y, m, perm, n, batch, (const float *)norm,
                                 (const float *)(norm + nin), p, m1, m2, loss, bc, lr, beta1, beta2, eps));
    c.launches++;
}

void Mlp::train(Ctx &c, const float *X, const float *T, const float *M, int n, int epochs, int batch, float lr,
                uint64_t seed, float *loss_hist) {
    if (n < 1 || epochs < 1 || batch < 1) throw CudaError{"invalid training arguments"};
    batch = std::min(batch, n);
    const EpochNet net{nin, hid, nout};
    const int np = (int)nparams();
    const bool fused = np <= kEpochParams && net.bytes(batch) <= kEpochSmem;
    if (fused) SAGB_CUDA(cudaFuncSetAttribute(k_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEpochSmem));
    else reserve(batch);
    load(c, X, T, M, n);
    const int steps_per_epoch = (n + batch - 1) / batch;
    // row orders, bias corrections and losses of some epochs
    const int chunk = std::min(epochs, std::max(1, kTrainRows / n));
    const size_t need = (size_t)chunk * ((size_t)n + 3 * (size_t)steps_per_epoch);
    if (need > train_cap) {
        dfree(perm_d);
        perm_d = nullptr;
        train_cap = 0;
        perm_d = (int *)dmalloc(need * sizeof(int));
        train_cap = need;
    }
    float2 *bc_d = (float2 *)perm_d;
    int *order_d = perm_d + 2 * (size_t)chunk * steps_per_epoch;
    float *dloss = (float *)(order_d + (size_t)chunk * n);
    std::vector<int> host((size_t)chunk * (2 * (size_t)steps_per_epoch + n));
    std::vector<float> ep_loss((size_t)chunk * steps_per_epoch);
    uint64_t st = seed;
    auto next = [&]() {
        uint64_t z = (st += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    for (int e0 = 0; e0 < epochs; e0 += chunk) {
        const int ne = std::min(chunk, epochs - e0);
        float2 *bc = (float2 *)host.data();
        int *order = host.data() + 2 * (size_t)chunk * steps_per_epoch;
        for (int e = 0; e < ne; e++) {
            int *perm = order + (size_t)e * n;
            for (int i = 0; i < n; i++) perm[i] = i;
            for (int i = n - 1; i > 0; i--) std::swap(perm[i], perm[next() % (uint64_t)(i + 1)]);  // Fisher-Yates
            for (int s = 0; s < steps_per_epoch; s++) {
                t++;
                bc[(size_t)e * steps_per_epoch + s] = make_float2(1.f - std::pow(beta1, (float)t), 1.f - std::pow(beta2, (float)t));
            }
        }
        SAGB_CUDA(cudaMemcpyAsync(perm_d, host.data(), host.size() * sizeof(int), cudaMemcpyHostToDevice, c.stream));
        for (int e = 0; e < ne; e++) {
            const int *perm = order_d + (size_t)e * n;
            const size_t s0 = (size_t)e * steps_per_epoch;
            if (fused) {
                launch_epoch(c, net, perm, n, batch, dloss + s0, bc_d + s0, lr, beta1, beta2, eps);
                continue;
            }
            for (int s = 0; s < steps_per_epoch; s++) {
                const int off = s * batch, B = std::min(batch, n - off);
                gather(c, perm, off, B, true);
                forward_batch(c, B);
                backward_batch(c, B);
                SAGB_CUDA(cudaMemcpyAsync(dloss + s0 + s, loss_slot(), sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
                const float2 k = bc[s0 + s];
                k_adam<<<(np + 255) / 256, 256, 0, c.stream>>>(p, g, m1, m2, np, lr, beta1, beta2, eps, k.x, k.y);
                c.launches++;
            }
        }
        SAGB_CUDA(cudaMemcpyAsync(ep_loss.data(), dloss, (size_t)ne * steps_per_epoch * sizeof(float),
                                  cudaMemcpyDeviceToHost, c.stream));
        SAGB_CUDA(cudaStreamSynchronize(c.stream));  // the host arrays are reused
        for (int e = 0; loss_hist && e < ne; e++) {
            float sum = 0.f;
            for (int k = 0; k < steps_per_epoch; k++) sum += ep_loss[(size_t)e * steps_per_epoch + k];
            loss_hist[e0 + e] = sum / steps_per_epoch;
        }
    }
}

void Mlp::get_params(float *out) const {
    SAGB_CUDA(cudaMemcpy(out, p, nparams() * sizeof(float), cudaMemcpyDeviceToHost));
}

void Mlp::set_params(const float *in) {
    SAGB_CUDA(cudaMemcpy(p, in, nparams() * sizeof(float), cudaMemcpyHostToDevice));
    SAGB_CUDA(cudaMemset(m1, 0, 2 * nparams() * sizeof(float)));
    t = 0;
}

}  // namespace sagb
