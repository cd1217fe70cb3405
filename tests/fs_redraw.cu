// Draws of a Fiat-Shamir transcript (truepix_b200/csrc/transcript.cuh) on the host and by
// a warp of the device, compiled with a bound that most draws miss.
#include "../truepix_b200/csrc/transcript.cuh"

using tp::fs::State;

namespace {

struct Draws {
    int count;
    tp::fs::Label label;
};

// puts between the draws: one element more each time, so that draws start at many offsets
__global__ void draw_kernel(State* st, Draws d, ulonglong2* out)
{
    __shared__ tp::fs::TxMem mem;
    tp::fs::Writer s(st[blockIdx.x], &mem);
    for (int k = 0; k < d.count; ++k) {
        for (int j = 0; j < k; ++j) s.put_fp2(1000 + k, j);
        const tp::fp2 r = s.rand_fp2(d.label);
        if (tp::fs::lead()) out[blockIdx.x * d.count + k] = make_ulonglong2(r.re, r.im);
    }
    s.store(st[blockIdx.x]);
}

Draws draws(int count, const char* label)
{
    Draws d = {count, {}};
    for (; *label; ++label) tp::fs::label_push(d.label, (uint8_t)*label);
    return d;
}

}  // namespace

extern "C" {

// n states of `each` put bytes more than the one before
void redraw_start(State* st, int n, int each)
{
    for (int i = 0; i < n; ++i) {
        tp::fs::init(st[i]);
        for (int j = 0; j < 64 + each * i; ++j) tp::fs::absorb_byte(st[i], (uint8_t)(7 * j + 3));
    }
}

void redraw_host(State* st, int n, int count, const char* label, ulonglong2* out)
{
    const Draws d = draws(count, label);
    for (int i = 0; i < n; ++i)
        for (int k = 0; k < count; ++k) {
            for (int j = 0; j < k; ++j) tp::fs::put_fp2(st[i], 1000 + k, j);
            const tp::fp2 r = tp::fs::rand_fp2(st[i], d.label);
            out[i * count + k] = make_ulonglong2(r.re, r.im);
        }
}

int redraw_device(State* st, int n, int count, const char* label, ulonglong2* out)
{
    State* d_st = nullptr;
    ulonglong2* d_out = nullptr;
    bool ok = cudaMalloc(&d_st, sizeof(State) * n) == cudaSuccess &&
              cudaMalloc(&d_out, sizeof(ulonglong2) * n * count) == cudaSuccess &&
              cudaMemcpy(d_st, st, sizeof(State) * n, cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) {
        draw_kernel<<<n, 32>>>(d_st, draws(count, label), d_out);
        ok = cudaGetLastError() == cudaSuccess &&
             cudaMemcpy(st, d_st, sizeof(State) * n, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(out, d_out, sizeof(ulonglong2) * n * count, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(d_st);
    cudaFree(d_out);
    return ok ? 0 : -1;
}

int redraw_state_bytes() { return (int)sizeof(State); }

}  // extern "C"
