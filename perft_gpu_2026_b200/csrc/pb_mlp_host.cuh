// pb_mlp_host.cuh - host side of the learned scheduler's network: parameter
// layout, initialisation, training loop (Adam) and inference.
//
// Flat FP32 parameter layout (also the layout of pb_mlp_get/set_params):
//   [ W1 781x256 | b1 256 | W2 256x256 | b2 256 | W3 256x4 | b3 4 ]
// W1 rows are input features, W2[i][j] maps hidden-1 unit i to hidden-2
// unit j, W3[j][o] maps hidden-2 unit j to output o.
#pragma once
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "pb_mlp.cuh"
#include "pb_util.cuh"

namespace pb {

constexpr size_t MLP_OFF_W1 = 0;
constexpr size_t MLP_OFF_B1 = MLP_OFF_W1 + (size_t)MLP_IN * MLP_H;
constexpr size_t MLP_OFF_W2 = MLP_OFF_B1 + MLP_H;
constexpr size_t MLP_OFF_B2 = MLP_OFF_W2 + (size_t)MLP_H * MLP_H;
constexpr size_t MLP_OFF_W3 = MLP_OFF_B2 + MLP_H;
constexpr size_t MLP_OFF_B3 = MLP_OFF_W3 + (size_t)MLP_H * MLP_OUT;
constexpr size_t MLP_PARAMS = MLP_OFF_B3 + MLP_OUT;

struct Mlp {
    bool ready = false;
    int max_batch = 0;
    u64 step = 0;
    // parameters, gradients, Adam moments (FP32) and the BF16 copy
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16 *pb = nullptr;
    // activations for one batch
    int16_t *idx = nullptr;
    float *h1f = nullptr, *z2 = nullptr, *h2f = nullptr, *y = nullptr, *dy = nullptr, *parts = nullptr,
          *dh1 = nullptr, *t = nullptr, *loss = nullptr;
    u32 *err = nullptr;     // GEMM error word (a tensor-core wait that gave up)
    float *work = nullptr;  // GEMM K-split partial tiles
    static constexpr size_t WORK_ELEMS = (size_t)tc::MAX_SPLITS * MLP_H * MLP_H;
    __nv_bfloat16 *h1b = nullptr, *dh2b = nullptr;
    PosBytes *pos = nullptr;
    // The training set of the last mlp_train (a piece of positions, feature indices,
    // targets, order, losses of an epoch's steps), kept for the next one unless
    // larger than TRAIN_KEEP: allocating and freeing it took 0.4 ms per call.
    char *train = nullptr;
    size_t train_bytes = 0;
    static constexpr size_t TRAIN_KEEP = (size_t)64 << 20;

    void release()
    {
        void *ptrs[] = {p,  g,     m,   v, pb,   idx, h1f,  z2,  h2f, y,
                        dy, parts, dh1, t, loss, err, work, h1b, dh2b, pos, train};
        for (void *q : ptrs)
            if (q) cudaFree(q);
        *this = Mlp();
    }

    // Device arrays of a training run over n examples and `steps` steps.
    struct TrainSet {
        PosBytes *pos;
        int16_t *idx;
        float *t;
        int *order;
        float *losses;
    };
    cudaError_t alloc_train(size_t n, size_t steps, TrainSet *set)
    {
        size_t off[6] = {0};
        const size_t bytes[5] = {std::min<size_t>(n, FEATURE_PIECE) * sizeof(PosBytes), n * MLP_MAX_ACTIVE * sizeof(int16_t),
                                 n * MLP_OUT * sizeof(float), n * sizeof(int), steps * sizeof(float)};
        for (int k = 0; k < 5; k++) off[k + 1] = off[k] + ((bytes[k] + 255) & ~(size_t)255);
        if (off[5] > train_bytes) {
            if (train) cudaFree(train);
            train = nullptr;
            train_bytes = 0;
            cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&train), off[5]);
            if (e != cudaSuccess) return e;
            train_bytes = off[5];
        }
        set->pos = reinterpret_cast<PosBytes *>(train + off[0]);
        set->idx = reinterpret_cast<int16_t *>(train + off[1]);
        set->t = reinterpret_cast<float *>(train + off[2]);
        set->order = reinterpret_cast<int *>(train + off[3]);
        set->losses = reinterpret_cast<float *>(train + off[4]);
        return cudaSuccess;
    }
    void trim_train()
    {
        if (train_bytes <= TRAIN_KEEP) return;
        cudaFree(train);
        train = nullptr;
        train_bytes = 0;
    }

    cudaError_t alloc_batch(int B)
    {
        if (B <= max_batch) return cudaSuccess;
        void *old[] = {idx, h1f, z2, h2f, y, dy, parts, dh1, t, h1b, dh2b, pos};
        for (void *q : old)
            if (q) cudaFree(q);
        cudaError_t e;
        size_t H = (size_t)B * MLP_H;
#define PB_MLP_ALLOC(ptr, bytes) \
    if ((e = cudaMalloc(reinterpret_cast<void **>(&ptr), bytes)) != cudaSuccess) return e;
        PB_MLP_ALLOC(idx, (size_t)B * MLP_MAX_ACTIVE * sizeof(int16_t));
        PB_MLP_ALLOC(h1f, H * 4);
        PB_MLP_ALLOC(z2, H * 4);
        PB_MLP_ALLOC(h2f, H * 4);
        PB_MLP_ALLOC(parts, (size_t)(B + BACK_SAMPLES - 1) / BACK_SAMPLES * BACK_PARTS * 4);
        PB_MLP_ALLOC(dh1, H * 4);
        PB_MLP_ALLOC(h1b, H * 2);
        PB_MLP_ALLOC(dh2b, H * 2);
        PB_MLP_ALLOC(y, (size_t)B * MLP_OUT * 4);
        PB_MLP_ALLOC(dy, (size_t)B * MLP_OUT * 4);
        PB_MLP_ALLOC(t, (size_t)B * MLP_OUT * 4);
        PB_MLP_ALLOC(pos, (size_t)std::min(B, FEATURE_PIECE) * sizeof(PosBytes));
#undef PB_MLP_ALLOC
        max_batch = B;
        return cudaSuccess;
    }

    // He-uniform weights from a splitmix64 stream, zero biases (b3 = out_bias).
    cudaError_t init(u64 seed, const float *out_bias, cudaStream_t s)
    {
        release();
        cudaError_t e;
        size_t bytes = MLP_PARAMS * sizeof(float);
        if ((e = cudaMalloc(&p, bytes)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&g, bytes)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&m, bytes)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&v, bytes)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&pb, MLP_PARAMS * sizeof(__nv_bfloat16))) != cudaSuccess) return e;
        if ((e = cudaMalloc(&loss, 64)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&err, sizeof(u32))) != cudaSuccess) return e;
        if ((e = cudaMalloc(&work, WORK_ELEMS * sizeof(float))) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(err, 0, sizeof(u32), s)) != cudaSuccess) return e;
        std::vector<float> h(MLP_PARAMS, 0.f);
        u64 st = seed;
        auto uni = [&](float lim) {
            u64 r = splitmix64(&st);
            return lim * (2.0f * (float)((r >> 11) * (1.0 / 9007199254740992.0)) - 1.0f);
        };
        // layer 1 sees ~35 active inputs of 781, so scale by the active fan-in
        float l1 = sqrtf(6.f / 35.f), l2 = sqrtf(6.f / MLP_H), l3 = sqrtf(3.f / MLP_H);
        for (size_t i = 0; i < (size_t)MLP_IN * MLP_H; i++) h[MLP_OFF_W1 + i] = uni(l1);
        for (size_t i = 0; i < (size_t)MLP_H * MLP_H; i++) h[MLP_OFF_W2 + i] = uni(l2);
        for (size_t i = 0; i < (size_t)MLP_H * MLP_OUT; i++) h[MLP_OFF_W3 + i] = uni(l3);
        if (out_bias)
            for (int o = 0; o < MLP_OUT; o++) h[MLP_OFF_B3 + o] = out_bias[o];
        if ((e = set_params(h.data(), s)) != cudaSuccess) return e;
        step = 0;
        ready = true;
        return cudaSuccess;
    }

    cudaError_t set_params(const float *host, cudaStream_t s)
    {
        cudaError_t e;
        size_t bytes = MLP_PARAMS * sizeof(float);
        if ((e = cudaMemcpyAsync(p, host, bytes, cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(m, 0, bytes, s)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(v, 0, bytes, s)) != cudaSuccess) return e;
        k_to_bf16<<<(unsigned)((MLP_PARAMS + 255) / 256), 256, 0, s>>>(p, MLP_PARAMS, pb);
        step = 0;
        return cudaGetLastError();
    }

    // Feature indices of n positions into rows [0, n) of `out`, by way of `dev`
    // (room for n or FEATURE_PIECE positions) a piece at a time; rows up to `rows`
    // get none.  The pieces bound the device memory that positions take and keep
    // the kernel's 32-bit thread index (32 threads a row) in range.
    static constexpr int FEATURE_PIECE = 1 << 20;
    static_assert((u64)FEATURE_PIECE * 32 + 256 <= 0xFFFFFFFFu, "thread indices of a piece fit 32 bits");
    cudaError_t features_to(const pb_pos *from, PosBytes *dev, int n, int rows, int16_t *out, cudaStream_t s)
    {
        static_assert(sizeof(pb_pos) == sizeof(PosBytes), "positions are copied as they are");
        for (size_t first = 0; first < (size_t)rows; first += FEATURE_PIECE) {
            const int r = (int)std::min<size_t>((size_t)rows - first, FEATURE_PIECE);
            const int k = (int)std::min<size_t>(r, (size_t)n - std::min((size_t)n, first));
            cudaError_t e = cudaSuccess;
            if (k) e = cudaMemcpyAsync(dev, from + first, sizeof(PosBytes) * k, cudaMemcpyHostToDevice, s);
            if (e != cudaSuccess) return e;
            k_features<<<(unsigned)(((size_t)r * 32 + 255) / 256), 256, 0, s>>>(dev, k, r, out + first * MLP_MAX_ACTIVE);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    // A batch: feature indices and targets by row, the batch's samples by `order`
    // (null: rows 0, 1, ...).
    struct Batch {
        const int16_t *idx;
        const float *t;    // null: forward only
        const int *order;
        float *loss;       // squared error sum, added to
    };

    // Forward over B samples (a multiple of 64); with targets also the loss, its
    // gradient and all parameter gradients.  dW1 and db1 are added to `g` (zeroed
    // by the caller, then by every adam_step).
    cudaError_t forward_backward(int B, const Batch &in, cudaStream_t s)
    {
        const __nv_bfloat16 *w1 = pb + MLP_OFF_W1, *w2 = pb + MLP_OFF_W2, *w3 = pb + MLP_OFF_W3;
        k_mlp_layer1<<<(B + L1_SAMPLES - 1) / L1_SAMPLES, 64 * L1_SAMPLES, 0, s>>>(
            in.idx, in.order, w1, p + MLP_OFF_B1, B, in.t ? h1f : nullptr, h1b);
        cudaError_t e =
            gemm_tc<false, false>(h1b, MLP_H, w2, MLP_H, z2, MLP_H, B, MLP_H, MLP_H, err, work, WORK_ELEMS, s);
        if (e != cudaSuccess) return e;
        k_mlp_out<<<(B + 8 * OUT_SAMPLES - 1) / (8 * OUT_SAMPLES), 256, 0, s>>>(
            z2, p + MLP_OFF_B2, w3, p + MLP_OFF_B3, B, y, in.t, in.order, h2f, dy, in.loss);
        if (!in.t) return cudaGetLastError();
        const int np = (B + BACK_SAMPLES - 1) / BACK_SAMPLES;
        k_back_h2<<<np, MLP_H, 0, s>>>(dy, w3, h2f, B, dh2b, parts);
        k_sum_parts<<<(BACK_PARTS + 31) / 32, 256, 0, s>>>(parts, np, g + MLP_OFF_W3, g + MLP_OFF_B2,
                                                            g + MLP_OFF_B3);
        // dW2 = h1^T dh2 ; dh1 = dh2 W2^T
        if ((e = gemm_tc<true, false>(h1b, MLP_H, dh2b, MLP_H, g + MLP_OFF_W2, MLP_H, MLP_H, MLP_H, B, err, work,
                                      WORK_ELEMS, s)) != cudaSuccess)
            return e;
        if ((e = gemm_tc<false, true>(dh2b, MLP_H, w2, MLP_H, dh1, MLP_H, B, MLP_H, MLP_H, err, work, WORK_ELEMS,
                                      s)) != cudaSuccess)
            return e;
        k_back_l1<<<(B + 4 * BACK1_SAMPLES - 1) / (4 * BACK1_SAMPLES), 256, 0, s>>>(
            in.idx, in.order, dh1, h1f, B, g + MLP_OFF_W1, g + MLP_OFF_B1);
        return cudaGetLastError();
    }
    cudaError_t clear_gradients(cudaStream_t s)
    {
        return cudaMemsetAsync(g + MLP_OFF_W1, 0, sizeof(float) * (MLP_OFF_W2 - MLP_OFF_W1), s);
    }

    cudaError_t adam_step(float lr, cudaStream_t s)
    {
        const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
        step++;
        float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
        k_adam<<<(unsigned)((MLP_PARAMS + 255) / 256), 256, 0, s>>>(p, g, MLP_OFF_W2, m, v, pb, MLP_PARAMS, lr, b1, b2, eps,
                                                                    c1, c2);
        return cudaGetLastError();
    }
};

}  // namespace pb
