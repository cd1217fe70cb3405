// Host side of the early-round sessions: a Batch of frames advanced round by
// round, one kernel launch per round (per source kind) for all frames.
//
// State machine per frame (TruePix-main/native_fp2/native_fp2_core.hpp:163-298
// for the single-session semantics): claim() evaluates the round polynomial at
// 0, 1, -1, 2 over the current copies; fold(r) records r and is applied by the
// next claim in the same pass (fold + claim fused), by a second fold, or by
// finish(). The first table of a frame may be its uint8 bytes; it is then
// never materialised.
#include "gkr.h"
#include "gkr_internal.cuh"
#include "runtime.h"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

namespace tp {

namespace {

// (re)use the frame's buffers: grow only when a configuration needs more. The frame
// counts as loaded once its loader has put everything in place, not before.
bool frame_alloc(Frame* f, size_t rows0, size_t rows1, cudaStream_t s)
{
    const size_t n = (size_t)f->n_copies0;
    if (f->borrowed0) {
        f->buf[0] = nullptr;
        f->cap0 = 0;
        f->borrowed0 = false;
    }
    if (rows0 > f->cap0) {
        dev_free(f->buf[0], s);
        f->buf[0] = (fp2*)dev_alloc(sizeof(fp2) * rows0, s);
        f->cap0 = f->buf[0] ? rows0 : 0;
    }
    if (rows1 > f->cap1) {
        dev_free(f->buf[1], s);
        f->buf[1] = (fp2*)dev_alloc(sizeof(fp2) * rows1, s);
        f->cap1 = f->buf[1] ? rows1 : 0;
    }
    if (n > f->capb) {
        dev_free(f->beta[0], s);
        dev_free(f->beta[1], s);
        f->beta[0] = (fp2*)dev_alloc(sizeof(fp2) * n, s);
        f->beta[1] = (fp2*)dev_alloc(sizeof(fp2) * n, s);
        f->capb = (f->beta[0] && f->beta[1]) ? n : 0;
    }
    f->cur = 0;
    f->pending = false;
    f->r_dev = nullptr;
    f->pix_cur = false;
    f->linear = f->loaded = false;
    return (!rows0 || f->buf[0]) && (!rows1 || f->buf[1]) && f->beta[0] && f->beta[1];
}

template <class T>
bool grow(T*& p, size_t& cap, size_t n, cudaStream_t s)
{
    if (n <= cap) return true;
    dev_free(p, s);
    p = static_cast<T*>(dev_alloc(sizeof(T) * n, s));
    cap = p ? n : 0;
    return p != nullptr;
}

// Whether a byte frame's rounds run on vectors (gkr_linear.cu): 1 + 2 groups vectors in
// place of W_rows rows. A round moves so many times less, against a pass over the bytes
// for every group and one more at the end. 384 bytes a copy, one frame, a call a round,
// rows -> vectors in us: no group, 2 copies 46 -> 54, 4 copies 70 -> 67, 8,192 copies
// 271 -> 198; one group 182 -> 168 and 456 -> 313; 4 groups 255 -> 250 and 538 -> 448;
// 8 groups 281 -> 291, 552 -> 552, and from 16,384 copies on 673 -> 592.
// A frame given as a table stays on its rows: its vectors cost two passes over 16 bytes a
// wire and won nothing in the same rounds (512 wires: 32 copies 98 -> 118, 2,048 copies
// 203 -> 196, 8,192 copies 319 -> 329; 16 wires and 32,768 copies 246 -> 582; 2^18 wires
// and 2 copies 0.8 -> 17 ms).
bool wants_linear(const Frame* f)
{
    const int G = f->form.groups;
    return f->n_copies0 >= 4 && G <= kMaxLinGroups && 4 * (1 + 2 * G) <= f->W_rows &&
           (G <= 4 || f->n_copies0 >= 2048 * G);
}

// the vectors' buffers of a frame; `part`: elements of the finish's scratch
bool linear_alloc(Frame* f, size_t part, cudaStream_t s)
{
    const size_t C = (size_t)f->n_copies0, nv = 1 + 2 * (size_t)f->form.groups;
    // one block: vectors of C copies, then of C / 2
    fp2* base = f->vec[0];
    if (!grow(base, f->capv, nv * C + nv * std::max<size_t>(1, C / 2), s)) {
        f->vec[0] = nullptr;
        return false;
    }
    f->vec[0] = base;
    f->vec[1] = base + nv * C;
    if (!f->rs) f->rs = static_cast<fp2*>(dev_alloc(sizeof(fp2) * 128, s));
    f->linear = true;
    f->forms_done = false;
    f->folds = 0;
    return f->rs && grow(f->fpart, f->cap_part, part, s);
}

void linear_free(Frame* f, cudaStream_t s)
{
    dev_free(f->vec[0], s);
    dev_free(f->bytes, s);
    dev_free(f->fpart, s);
    f->vec[0] = f->vec[1] = f->fpart = nullptr;
    f->bytes = nullptr;
    f->capv = f->cap_bytes = f->cap_part = 0;
}

// apply a recorded fold without a claim
bool apply_fold(Frame* f, cudaStream_t s, int* launches)
{
    const int n_out = f->n_phys >> 1;
    if (f->pix_cur) {
        if (!launch_fold_pixels(f->px, f->W_rows, n_out, f->r, f->buf[1], f->beta[0], f->beta[1], s,
                                launches))
            return false;
        f->pix_cur = false;
        f->cur = 1;
    } else {
        const int nxt = f->cur ^ 1;
        if (!launch_fold_rows(f->buf[f->cur], f->n_phys, f->buf[nxt], f->W_rows, f->beta[f->cur],
                              f->beta[nxt], f->r, s, launches))
            return false;
        f->cur = nxt;
    }
    f->n_phys = n_out;
    f->pending = false;
    return true;
}

bool ensure_workspace(Batch* B, size_t jobs, size_t ctas)
{
    cudaStream_t s = B->stream;
    if (jobs > B->cap_jobs) {
        dev_free(B->d_jobs, s);
        B->cap_jobs = std::max<size_t>(jobs, 16);
        B->d_jobs = (Job*)dev_alloc(sizeof(Job) * B->cap_jobs, s);
        if (!B->d_jobs) return false;
    }
    if (jobs > B->cap_tickets) {
        dev_free(B->tickets, s);
        B->cap_tickets = std::max<size_t>(jobs, 16);
        B->tickets = (unsigned*)dev_alloc(sizeof(unsigned) * B->cap_tickets, s);
        if (!B->tickets) return false;
        TP_CUDA_OK(cudaMemsetAsync(B->tickets, 0, sizeof(unsigned) * B->cap_tickets, s), "tickets");
    }
    if (ctas > B->cap_partials) {
        dev_free(B->partials, s);
        B->cap_partials = std::max<size_t>(ctas, 4096);
        B->partials = (fp2*)dev_alloc(sizeof(fp2) * 4 * B->cap_partials, s);
        if (!B->partials) return false;
    }
    return true;
}

// A job whose frame's pending fold takes its challenge from device memory gets
// it written into the uploaded job array, in stream order, before the launch.
struct RPatch {
    const fp2* r;
    long long job;
};

__global__ void patch_r_kernel(Job* __restrict__ jobs, const RPatch* __restrict__ p, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) jobs[p[i].job].r = *p[i].r;
}

bool upload_jobs(Batch* B, const Job* jobs, size_t n, const std::vector<const fp2*>& rdev)
{
    if (!upload_async(B->d_jobs, jobs, sizeof(Job) * n, B->stream)) return false;
    std::vector<RPatch> p;
    for (size_t q = 0; q < n && q < rdev.size(); ++q)
        if (rdev[q]) p.push_back(RPatch{rdev[q], (long long)q});
    if (p.empty()) return true;
    if (p.size() > B->cap_patch) {
        dev_free(B->d_patch, B->stream);
        B->cap_patch = std::max<size_t>(p.size(), 64);
        B->d_patch = dev_alloc(sizeof(RPatch) * B->cap_patch, B->stream);
        if (!B->d_patch) {
            B->cap_patch = 0;
            return false;
        }
    }
    if (!upload_async(B->d_patch, p.data(), sizeof(RPatch) * p.size(), B->stream)) return false;
    patch_r_kernel<<<(unsigned)((p.size() + 127) / 128), 128, 0, B->stream>>>(
        B->d_jobs, static_cast<const RPatch*>(B->d_patch), (int)p.size());
    ++B->launches;
    return !cuda_failed(cudaGetLastError(), "challenge patch");
}

bool device_fold_blocked(const Frame* f)
{
    if (f->pending && f->r_dev) {
        set_error(TP_ERR_ARG, "a fold with a device challenge needs a claim or finish before the next fold");
        return true;
    }
    return false;
}

Job base_job(const Frame* f)
{
    Job j;
    memset(&j, 0, sizeof(j));
    j.L = f->form.L;
    j.ab = f->form.ab;
    j.cf = f->form.c;
    j.n_terms = f->form.n_terms;
    j.K0 = f->form.K0;
    j.Lc = f->Lc;
    j.r = f->r;
    j.W = f->n_wires;
    j.W_rows = f->W_rows;
    j.n_in = f->n_phys;
    j.beta = f->beta[f->cur];
    if (f->linear) {
        j.A = f->vec[f->cur];
        j.Aout = f->vec[f->cur ^ 1];
        j.beta_out = f->beta[f->cur ^ 1];
        j.G = f->form.groups;
        j.gptr = f->form.gptr;
        j.gb = f->form.gb;
        j.rs = f->rs;
        j.given = f->rs + 64;
        j.nf = f->folds;
        j.has_r = f->pending ? 1 : 0;
        j.fpart = f->fpart;
        j.pix = f->px.pix;
        j.n_real = f->px.n_real;
        j.cs = f->px.cs;
        j.const_idx = f->px.const_idx;
        j.const_val = f->px.const_val;
        j.bytes = f->bytes;
        j.stride = lin_stride(f->px.cs);
        j.chunks = lin_chunks(f->px.n_real, f->folds + j.has_r);
        j.vec = ((j.cs & 15) == 0 && (reinterpret_cast<size_t>(j.pix) & 15) == 0) ? 1 : 0;
    } else if (f->pix_cur) {
        j.pix = f->px.pix;
        j.n_real = f->px.n_real;
        j.cs = f->px.cs;
        j.const_idx = f->px.const_idx;
        j.const_val = f->px.const_val;
    } else {
        j.A = f->buf[f->cur];
    }
    return j;
}

// the fold that a claim launch applies has been planned into it
void advance_fold(Frame* f)
{
    f->cur = f->pix_cur ? 1 : (f->cur ^ 1);
    f->pix_cur = false;
    f->n_phys >>= 1;
    f->pending = false;
    f->r_dev = nullptr;
    if (f->linear) ++f->folds;
}

}  // namespace

Batch* batch_create(int n_frames, cudaStream_t s)
{
    if (n_frames <= 0) {
        set_error(TP_ERR_ARG, "a batch needs at least one frame");
        return nullptr;
    }
    if (!ctx()) return nullptr;
    Batch* B = new Batch();
    B->stream = s;
    for (int i = 0; i < n_frames; ++i) B->frames.push_back(new Frame());
    return B;
}

namespace {

// frame i's shape and its form on the host; finish_set_gates follows once the form
// has its place on the device
bool start_set_gates(Batch* B, int i, int n_gates, const int* type, const int* in0, const int* in1, const u64* z_re,
                     const u64* z_im, int n_copies, int n_wires, GateForm& g)
{
    if (i < 0 || i >= (int)B->frames.size()) {
        set_error(TP_ERR_ARG, "frame index %d outside the batch", i);
        return false;
    }
    if (n_gates <= 0 || n_wires <= 0 || n_copies < 2 || (n_copies & (n_copies - 1)) != 0) {
        set_error(TP_ERR_ARG, "early session needs n_gates > 0, n_wires > 0 and n_copies a "
                              "power of two >= 2 (got %d, %d, %d)", n_gates, n_wires, n_copies);
        return false;
    }
    Frame* f = B->frames[(size_t)i];
    if (f->configured) {
        set_error(TP_ERR_ARG, "frame %d is already configured (tp_batch_reset first)", i);
        return false;
    }
    if (!build_gate_form(n_gates, type, in0, in1, z_re, z_im, n_wires, g)) return false;
    f->loaded = false;
    f->n_wires = f->W_rows = n_wires;
    f->n_copies0 = f->n_copies = f->n_phys = n_copies;
    f->L_host = g.L;
    f->Lc = f2zero();
    return true;
}

bool finish_set_gates(Batch* B, Frame* f)
{
    const int n_wires = f->n_wires;
    if ((size_t)n_wires + 1 > f->capfin) {
        dev_free(f->fin, B->stream);
        f->fin = (fp2*)dev_alloc(sizeof(fp2) * ((size_t)n_wires + 1), B->stream);
        f->capfin = f->fin ? (size_t)n_wires + 1 : 0;
    }
    if (!f->out8) f->out8 = (u64*)dev_alloc(64, B->stream);
    f->configured = f->fin && f->out8;
    return f->configured;
}

}  // namespace

bool batch_set_gates(Batch* B, int i, int n_gates, const int* type, const int* in0,
                     const int* in1, const u64* z_re, const u64* z_im, int n_copies, int n_wires)
{
    GateForm g;
    if (!start_set_gates(B, i, n_gates, type, in0, in1, z_re, z_im, n_copies, n_wires, g)) return false;
    Frame* f = B->frames[(size_t)i];
    return upload_gate_form(g, f->form, B->stream) && finish_set_gates(B, f);
}

bool batch_load_host(Batch* B, int i, const u64* v_re, const u64* v_im, const u64* b_re,
                     const u64* b_im)
{
    Frame* f = B->frames[(size_t)i];
    cudaStream_t s = B->stream;
    const size_t vn = (size_t)f->n_wires * (size_t)f->n_copies0;
    if (!frame_alloc(f, vn, vn / 2, s)) return false;
    // stage the real limbs in the half-size buffer (exactly vn u64), the
    // imaginary limbs in a temporary, then pack
    u64* stage_re = reinterpret_cast<u64*>(f->buf[1]);
    u64* stage_im = (u64*)dev_alloc(sizeof(u64) * vn, s);
    if (!stage_im) return false;
    int launches = 0;
    bool ok = host_to_device(stage_re, v_re, 8 * vn, s) && host_to_device(stage_im, v_im, 8 * vn, s) &&
              launch_pack(stage_re, stage_im, vn, f->buf[0], s, &launches);
    const size_t n = (size_t)f->n_copies0;
    u64* bst = reinterpret_cast<u64*>(f->beta[1]);  // 16 B x n: room for both limb arrays
    ok = ok && !cuda_failed(cudaMemcpyAsync(bst, b_re, 8 * n, cudaMemcpyHostToDevice, s), "H2D beta") &&
         !cuda_failed(cudaMemcpyAsync(bst + n, b_im, 8 * n, cudaMemcpyHostToDevice, s), "H2D beta") &&
         launch_pack(bst, bst + n, n, f->beta[0], s, &launches);
    B->launches += launches;
    dev_free(stage_im, s);
    // the reference contract: host inputs are consumed before the call returns
    f->loaded = ok && !cuda_failed(cudaStreamSynchronize(s), "load tables");
    return f->loaded;
}

bool batch_load_device(Batch* B, int i, const fp2* d_values, const fp2* d_beta, bool borrow)
{
    Frame* f = B->frames[(size_t)i];
    cudaStream_t s = B->stream;
    const size_t vn = (size_t)f->n_wires * (size_t)f->n_copies0;
    if (!frame_alloc(f, borrow ? 0 : vn, vn / 2, s)) return false;
    if (borrow) {
        f->buf[0] = const_cast<fp2*>(d_values);
        f->borrowed0 = true;
    } else {
        TP_CUDA_OK(cudaMemcpyAsync(f->buf[0], d_values, sizeof(fp2) * vn, cudaMemcpyDeviceToDevice, s),
                   "copy values");
    }
    TP_CUDA_OK(cudaMemcpyAsync(f->beta[0], d_beta, sizeof(fp2) * (size_t)f->n_copies0,
                               cudaMemcpyDeviceToDevice, s), "copy beta");
    f->loaded = true;
    return true;
}

namespace {

// everything of a byte frame but its copy of beta
bool start_load_pixels(Batch* B, int i, const PixSrc& px)
{
    Frame* f = B->frames[(size_t)i];
    if (!pixsrc_valid(px, f->n_copies0, f->n_wires)) return false;
    cudaStream_t s = B->stream;
    f->px = px;
    f->W_rows = pixsrc_rows(px);
    const size_t C = (size_t)f->n_copies0, R = (size_t)f->W_rows;
    if (wants_linear(f)) {
        if (!frame_alloc(f, 0, 0, s) || !linear_alloc(f, (size_t)lin_chunks(px.n_real, 30) * R, s) ||
            !grow(f->bytes, f->cap_bytes, lin_bytes(px.cs, px.n_real), s))
            return false;
    } else {
        // first fold writes R x C/2 into buf[1]; later folds alternate with buf[0]
        if (!frame_alloc(f, R * std::max<size_t>(1, C / 4), R * (C / 2), s)) return false;
        f->pix_cur = true;
    }
    if (px.const_idx >= 0) f->Lc = f2scale(f->L_host[(size_t)px.const_idx], px.const_val);
    return true;
}

struct BetaCopy {
    const fp2* src;
    fp2* dst;
    long long n;
};

__global__ void __launch_bounds__(256) copy_betas_kernel(const BetaCopy* __restrict__ list)
{
    const BetaCopy c = list[blockIdx.y];
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < c.n; i += (long long)gridDim.x * 256)
        st2(c.dst + i, ld2(c.src + i));
}

}  // namespace

bool batch_load_pixels(Batch* B, int i, const PixSrc& px, const fp2* d_beta)
{
    if (!start_load_pixels(B, i, px)) return false;
    Frame* f = B->frames[(size_t)i];
    TP_CUDA_OK(cudaMemcpyAsync(f->beta[0], d_beta, sizeof(fp2) * (size_t)f->n_copies0, cudaMemcpyDeviceToDevice,
                               B->stream),
               "copy beta");
    f->loaded = true;
    return true;
}

// One upload in a few pieces and one launch for all frames, where a call per frame made
// two copies and an event each (64 1080p frames: 1.98 ms of the host's time a proof, now
// 1.03). A beta that 16-byte loads cannot read is copied by itself.
bool batch_set_pixels_all(Batch* B, int n_gates, const int* type, const int* in0, const int* in1, const u64* z1,
                          const PixSrc* px, const int* n_copies, int n_wires, const fp2* const* d_betas)
{
    cudaStream_t s = B->stream;
    const int n = (int)B->frames.size();
    std::vector<unsigned char> h;
    std::vector<BetaCopy> betas;
    for (int i = 0; i < n; ++i) {
        if (B->frames[(size_t)i]->configured) {   // in the middle of its rounds, perhaps: the batch stays as it is
            set_error(TP_ERR_ARG, "frame %d is already configured (tp_batch_reset first)", i);
            return false;
        }
        if (!d_betas[i]) {
            set_error(TP_ERR_ARG, "frame %d has no beta", i);
            return false;
        }
    }
    auto aligned = [&](int i) { return (reinterpret_cast<size_t>(d_betas[i]) & 15) == 0; };
    auto all = [&]() -> bool {
        int most = 0;
        for (int i = 0; i < n; ++i) {
            Frame* f = B->frames[(size_t)i];
            const u64* z = z1 + (size_t)i * 2 * (size_t)n_gates;
            GateForm g;
            if (!start_set_gates(B, i, n_gates, type, in0, in1, z, z + n_gates, n_copies[i], n_wires, g)) return false;
            pack_gate_form(g, f->form, h);
            if (!finish_set_gates(B, f) || !start_load_pixels(B, i, px[i])) return false;
            betas.push_back(BetaCopy{d_betas[i], f->beta[0], aligned(i) ? n_copies[i] : 0});
            most = std::max(most, n_copies[i]);
        }
        h.resize((h.size() + 15) & ~(size_t)15);
        const size_t at = h.size();
        h.resize(at + sizeof(BetaCopy) * betas.size());
        memcpy(h.data() + at, betas.data(), sizeof(BetaCopy) * betas.size());
        unsigned char* forms = static_cast<unsigned char*>(B->forms);
        if (!grow(forms, B->cap_forms, h.size(), s)) {
            B->forms = nullptr;
            return false;
        }
        B->forms = forms;
        for (Frame* f : B->frames) place_gate_form(f->form, forms);
        constexpr size_t kPiece = 256 * 1024;   // what the staging ring takes without a wait
        for (size_t o = 0; o < h.size(); o += kPiece)
            if (!upload_async(forms + o, h.data() + o, std::min(kPiece, h.size() - o), s)) return false;
        copy_betas_kernel<<<dim3((unsigned)std::max(1, std::min(64, (most + 255) / 256)), (unsigned)n), 256, 0, s>>>(
            reinterpret_cast<const BetaCopy*>(forms + at));
        ++B->launches;
        if (cuda_failed(cudaGetLastError(), "copy betas")) return false;
        for (int i = 0; i < n; ++i)
            if (!aligned(i) &&
                cuda_failed(cudaMemcpyAsync(B->frames[(size_t)i]->beta[0], d_betas[i], sizeof(fp2) * (size_t)n_copies[i],
                                            cudaMemcpyDeviceToDevice, s),
                            "copy beta"))
                return false;
        for (Frame* f : B->frames) f->loaded = true;
        return true;
    };
    if (all()) return true;
    batch_reset(B);   // no frame was set before, none is left half set
    return false;
}

namespace {

// ---- round planning ----------------------------------------------------------
// A round launch is planned on the host from the frames' state (which it then
// advances as the launch will), before anything is uploaded: the immediate path
// uploads and launches it at once, the graph path plans every round of a proof
// first and replays them from one device job table.

// work of a launch, for the autotuner's size buckets
int work_bucket(const std::vector<Job>& jobs, int kind)
{
    double total = 0;
    for (const Job& j : jobs)
        total += kind == kFormsBytes ? 0.5 * j.n_in * j.cs : (double)j.n_pairs * (kind < 2 ? j.W_rows : j.cs);
    int b = 0;
    while (b < 62 && (double)(1ull << (b + 1)) <= total) ++b;
    return b;
}

// The claim/fold launch split: a round launch of one kind spreads `target` CTAs
// over its jobs in proportion to their work (pair tiles x row groups,
// plan_job). The autotuner measures the target, as CTAs per SM, per (kind, work
// bucket) on the device and keeps the fastest; 4 per SM until it has.
constexpr int kTuneMults[] = {2, 3, 4, 6, 8, 12, 16};

// one planned launch: a round kind (0..3) or the finish (kind 4)
struct RoundLaunch {
    int kind = 0;
    std::vector<Job> jobs;
    std::vector<const fp2*> rdev;   // per job: the device challenge patched into it, or null
    int bucket = 0;
    int timer_tag = 0;
    int max_w = 0;                  // finish: the widest frame
};

struct TuneKey {
    int device, kind, bucket;
    bool operator<(const TuneKey& o) const
    {
        return device != o.device ? device < o.device : kind != o.kind ? kind < o.kind : bucket < o.bucket;
    }
};
std::map<TuneKey, int>& tune_table()
{
    static std::map<TuneKey, int> t;
    return t;
}
std::mutex& tune_mutex()
{
    static std::mutex m;
    return m;
}
bool g_tune_on = false;

bool tune_known(int kind, int bucket)
{
    Ctx* c = ctx();
    std::lock_guard<std::mutex> lk(tune_mutex());
    return tune_table().count(TuneKey{c ? c->device : 0, kind, bucket}) != 0;
}

int tuned_mult(int kind, int bucket)
{
    Ctx* c = ctx();
    std::lock_guard<std::mutex> lk(tune_mutex());
    auto it = tune_table().find(TuneKey{c ? c->device : 0, kind, bucket});
    return it == tune_table().end() ? 4 : it->second;
}

void plan_jobs(std::vector<Job>& jobs, int kind, int target)
{
    double total = 0;
    for (const Job& j : jobs) total += (double)j.n_pairs * (kind < 2 ? j.W_rows : j.cs);
    int cta = 0;
    for (Job& j : jobs) {
        const double w = (double)j.n_pairs * (kind < 2 ? j.W_rows : j.cs);
        plan_job(j, std::max(1, (int)(target * w / total + 0.5)));
        j.cta0 = cta;
        cta += j.tiles * j.groups;
    }
}

// the same for the launches of frames on vectors: only the forms from bytes have a
// split (copies per CTA) to choose
void plan_linear_jobs(std::vector<Job>& jobs, int kind, int target)
{
    double total = 0;
    for (const Job& j : jobs) total += j.n_in;
    int cta = 0;
    for (Job& j : jobs) {
        plan_linear_job(j, kind, std::max(1, (int)(target * (double)j.n_in / total + 0.5)));
        j.cta0 = cta;
        cta += j.tiles;
    }
}

void plan_launch(std::vector<Job>& jobs, int kind, int target)
{
    if (kind < 4) plan_jobs(jobs, kind, target);
    else plan_linear_jobs(jobs, kind, target);
}

// the tuner's kind of a launch (the forms from bytes stand for the byte claim they
// replace), or -1 for one without a split
int tune_kind(int kind) { return kind < 4 ? kind : kind == kFormsBytes ? 2 : -1; }

size_t launch_ctas(const std::vector<Job>& jobs)
{
    size_t n = 0;
    for (const Job& j : jobs) n += (size_t)j.tiles * j.groups;
    return n;
}

void set_workspace_ptrs(Batch* B, std::vector<Job>& jobs)
{
    for (size_t q = 0; q < jobs.size(); ++q) {
        jobs[q].partials = B->partials + 4 * (size_t)jobs[q].cta0;
        jobs[q].ticket = B->tickets + q;
    }
}

// the launch that makes the vectors of frames which have none yet; appended to out
void plan_forms(const std::vector<Frame*>& frames, std::vector<RoundLaunch>& out, int n_sm)
{
    RoundLaunch L;
    L.kind = kFormsBytes;
    int lg = 0;
    for (Frame* f : frames) {
        if (!f->linear || f->forms_done) continue;
        Job j = base_job(f);
        j.kind = kFormsBytes;
        L.jobs.push_back(j);
        L.rdev.push_back(nullptr);
        f->forms_done = true;
        lg = 0;
        while ((1 << lg) < f->n_copies0) ++lg;
    }
    if (L.jobs.empty()) return;
    L.bucket = work_bucket(L.jobs, kFormsBytes);
    plan_linear_jobs(L.jobs, kFormsBytes, tuned_mult(2, L.bucket) * n_sm);
    L.timer_tag = 1000 + lg;
    out.push_back(std::move(L));
}

constexpr int kKinds = 6;   // 0..3 on tables and bytes, kVecClaim, kVecFold

// the claim launches of one round: per kind, its jobs and the device challenges
// of their pending folds; advances the frames past the round's folds
bool plan_claims(Batch* B, u64* const* d_claims, std::vector<RoundLaunch>& out)
{
    Ctx* c = ctx();
    if (!c) return false;
    RoundLaunch by_kind[kKinds];
    std::vector<Frame*> fr[kKinds], fresh;
    for (int k = 0; k < kKinds; ++k) by_kind[k].kind = k;
    bool any = false;
    for (size_t i = 0; i < B->frames.size(); ++i) {
        Frame* f = B->frames[i];
        if (!f->configured) continue;
        if (!f->loaded) {
            set_error(TP_ERR_ARG, "frame %zu has no table", i);
            return false;
        }
        if (f->n_copies < 2) continue;
        any = true;
        if (f->linear && !f->forms_done) fresh.push_back(f);
        Job j = base_job(f);
        j.kind = f->linear ? (f->pending ? kVecFold : kVecClaim) : (f->pix_cur ? 2 : 0) + (f->pending ? 1 : 0);
        if (f->pending && !f->linear) {
            const int nxt = f->pix_cur ? 1 : (f->cur ^ 1);
            j.Aout = f->buf[nxt];
            j.beta_out = f->beta[nxt];
        }
        j.n_pairs = f->n_copies / 2;
        j.out8 = (d_claims && d_claims[i]) ? d_claims[i] : f->out8;
        by_kind[j.kind].jobs.push_back(j);
        by_kind[j.kind].rdev.push_back(f->pending ? f->r_dev : nullptr);
        fr[j.kind].push_back(f);
    }
    if (B->frames.size() == 1 && !any) {
        set_error(TP_ERR_ARG, "claim needs at least 2 copies (have %d)", B->frames[0]->n_copies);
        return false;
    }
    plan_forms(fresh, out, c->n_sm);
    for (int k = 0; k < kKinds; ++k) {
        RoundLaunch& L = by_kind[k];
        if (L.jobs.empty()) continue;
        if (k < 4) L.bucket = work_bucket(L.jobs, k);
        plan_launch(L.jobs, k, (k < 4 ? tuned_mult(k, L.bucket) : 4) * c->n_sm);
        int lg = 0;
        while ((1 << lg) < 2 * L.jobs[0].n_pairs) ++lg;
        L.timer_tag = (k < 4 ? 1000 * (k >> 1) : 0) + 100 * (k & 1) + lg;
        for (Frame* f : fr[k])
            if (f->pending) advance_fold(f);
        out.push_back(std::move(L));
    }
    return true;
}

bool launch_any(const Job* d_jobs, const RoundLaunch& L, cudaStream_t s, int* launches)
{
    return L.kind < 4 ? launch_round(d_jobs, L.jobs, L.kind, s, launches)
                      : launch_linear(d_jobs, L.jobs, L.kind, s, launches);
}

// time one round launch under each candidate split, keep the fastest for its
// (kind, bucket); the launches rerun the same jobs (a claim or fold + claim
// reads its source and rewrites the same outputs)
bool tune_launch(Batch* B, RoundLaunch& L)
{
    Ctx* c = ctx();
    cudaStream_t s = B->stream;
    float best_ms = 0;
    int best = 4;
    cudaEvent_t e0, e1;
    TP_CUDA_OK(cudaEventCreate(&e0), "tune event");
    TP_CUDA_OK(cudaEventCreate(&e1), "tune event");
    bool ok = true;
    for (int mult : kTuneMults) {
        std::vector<Job> jobs = L.jobs;
        plan_launch(jobs, L.kind, mult * c->n_sm);
        if (!ensure_workspace(B, jobs.size(), launch_ctas(jobs))) {
            ok = false;
            break;
        }
        set_workspace_ptrs(B, jobs);
        if (!upload_jobs(B, jobs.data(), jobs.size(), L.rdev)) {
            ok = false;
            break;
        }
        int dummy = 0;
        RoundLaunch tried;
        tried.kind = L.kind;
        tried.jobs = std::move(jobs);
        ok = launch_any(B->d_jobs, tried, s, &dummy);   // warm
        ok = ok && !cuda_failed(cudaEventRecord(e0, s), "tune event");
        for (int rep = 0; ok && rep < 3; ++rep) ok = launch_any(B->d_jobs, tried, s, &dummy);
        ok = ok && !cuda_failed(cudaEventRecord(e1, s), "tune event") &&
             !cuda_failed(cudaEventSynchronize(e1), "tune sync");
        if (!ok) break;
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (best_ms == 0 || ms < best_ms) {
            best_ms = ms;
            best = mult;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!ok) return false;
    {
        std::lock_guard<std::mutex> lk(tune_mutex());
        tune_table()[TuneKey{c->device, tune_kind(L.kind), L.bucket}] = best;
    }
    plan_launch(L.jobs, L.kind, best * c->n_sm);
    return true;
}

bool launch_planned(Batch* B, RoundLaunch& L)
{
    const int tk = tune_kind(L.kind);
    if (g_tune_on && tk >= 0 && !tune_known(tk, L.bucket) && !tune_launch(B, L)) return false;
    if (!ensure_workspace(B, L.jobs.size(), launch_ctas(L.jobs))) return false;
    set_workspace_ptrs(B, L.jobs);
    if (!upload_jobs(B, L.jobs.data(), L.jobs.size(), L.rdev)) return false;
    timer_begin(B->stream, L.timer_tag);
    const bool ok = launch_any(B->d_jobs, L, B->stream, &B->launches);
    timer_end(B->stream);
    return ok;
}

// a linear frame's recorded fold without a claim of the caller's: the claim launch
// that applies it, its claim left in the frame's own slot
bool apply_fold_linear(Batch* B, Frame* f)
{
    Ctx* c = ctx();
    if (!c) return false;
    std::vector<RoundLaunch> plan;
    plan_forms({f}, plan, c->n_sm);
    RoundLaunch L;
    L.kind = kVecFold;
    Job j = base_job(f);
    j.kind = kVecFold;
    j.n_pairs = f->n_phys / 4;
    j.out8 = f->out8;
    plan_linear_job(j, kVecFold, 1);
    L.jobs.push_back(j);
    L.rdev.push_back(f->r_dev);
    advance_fold(f);
    plan.push_back(std::move(L));
    for (RoundLaunch& q : plan)
        if (!launch_planned(B, q)) return false;
    return true;
}

// whether a linear frame's rounds that are left run in one CTA
bool few_left(const Frame* f)
{
    const long long pairs = f->n_copies / 2;
    return pairs <= kFusePairs && pairs * (1 + 2 * f->form.groups) <= kFuseEntries;
}

// Rounds of a linear frame whose challenges (device memory at its given[]) are all
// known: n_rounds claims, each followed by its fold, in one launch; the last fold
// stays recorded (host challenge `last`). Planned into L.
void plan_given(Frame* f, int n_rounds, u64* out8, fp2 last, RoundLaunch& L)
{
    Job j = base_job(f);
    j.kind = kVecFold;
    j.n_rounds = n_rounds;
    j.out8 = out8;
    j.tiles = j.groups = 1;
    L.kind = kVecFold;
    L.jobs.push_back(j);
    L.rdev.push_back(f->pending ? f->r_dev : nullptr);
    if (f->pending) advance_fold(f);
    for (int q = 0; q < n_rounds; ++q) {
        f->n_copies >>= 1;
        if (q + 1 < n_rounds) advance_fold(f);
    }
    f->pending = true;
    f->r = last;
    f->r_dev = nullptr;
}

}  // namespace

bool batch_given_rounds(Batch* B, int n_rounds, const u64* challenges, u64* d_claims)
{
    Frame* f = B->frames[0];
    for (int k = 0; k < n_rounds; ++k) {
        // from here on in one launch: few pairs left, two rounds or more to go
        const int left = n_rounds - k;
        if (f->configured && f->loaded && f->linear && d_claims && left > 1 && left <= 63 &&
            few_left(f) && (f->n_copies >> left) >= 1) {
            std::vector<fp2> r;
            for (int q = k; q < n_rounds; ++q) {
                r.push_back(mk(challenges[2 * q], challenges[2 * q + 1]));
                if (r.back().re >= P61 || r.back().im >= P61) {
                    set_error(TP_ERR_ARG, "fold challenge is not a canonical field element");
                    return false;
                }
            }
            Ctx* c = ctx();
            if (!c) return false;
            std::vector<RoundLaunch> plan;
            plan_forms({f}, plan, c->n_sm);
            for (RoundLaunch& L : plan)
                if (!launch_planned(B, L)) return false;
            RoundLaunch L;
            if (!upload_async(f->rs + 64, r.data(), sizeof(fp2) * r.size(), B->stream)) return false;
            plan_given(f, left, d_claims + 8 * (size_t)k, r.back(), L);
            return ensure_workspace(B, 1, 1) && upload_jobs(B, L.jobs.data(), 1, L.rdev) &&
                   launch_linear_rounds(B->d_jobs, 1, nullptr, 0, 8, B->stream, &B->launches);
        }
        u64* p = d_claims ? d_claims + 8 * (size_t)k : nullptr;
        if (!batch_claim(B, &p)) return false;
        if (!batch_fold(B, 0, mk(challenges[2 * k], challenges[2 * k + 1]))) return false;
    }
    return true;
}

bool batch_claim(Batch* B, u64* const* d_claims)
{
    std::vector<RoundLaunch> plan;
    if (!plan_claims(B, d_claims, plan)) return false;
    for (RoundLaunch& L : plan)
        if (!launch_planned(B, L)) return false;
    return true;
}

bool batch_fold(Batch* B, int i, fp2 r)
{
    if (i < 0 || i >= (int)B->frames.size()) {
        set_error(TP_ERR_ARG, "frame index %d outside the batch", i);
        return false;
    }
    Frame* f = B->frames[(size_t)i];
    if (f->n_copies < 2) {
        set_error(TP_ERR_ARG, "fold needs at least 2 copies (have %d)", f->n_copies);
        return false;
    }
    if (r.re >= P61 || r.im >= P61) {
        set_error(TP_ERR_ARG, "fold challenge is not a canonical field element");
        return false;
    }
    if (device_fold_blocked(f)) return false;
    if (f->pending && !f->loaded) {
        set_error(TP_ERR_ARG, "frame %d has no table", i);
        return false;
    }
    if (f->pending && !(f->linear ? apply_fold_linear(B, f) : apply_fold(f, B->stream, &B->launches))) return false;
    f->pending = true;
    f->r = r;
    f->r_dev = nullptr;
    f->n_copies >>= 1;
    return true;
}

bool batch_fold_dev(Batch* B, int i, const fp2* d_r)
{
    if (i < 0 || i >= (int)B->frames.size()) {
        set_error(TP_ERR_ARG, "frame index %d outside the batch", i);
        return false;
    }
    Frame* f = B->frames[(size_t)i];
    if (f->n_copies < 2) {
        set_error(TP_ERR_ARG, "fold needs at least 2 copies (have %d)", f->n_copies);
        return false;
    }
    if (!d_r) {
        set_error(TP_ERR_ARG, "null device challenge");
        return false;
    }
    if (f->pending) {
        set_error(TP_ERR_ARG, "a fold with a device challenge needs a claim or finish after the previous fold");
        return false;
    }
    f->pending = true;
    f->r = f2zero();
    f->r_dev = d_r;
    f->n_copies >>= 1;
    return true;
}

namespace {

// The finish launches: wires and beta of every configured frame (a pending fold of
// the last two copies applied by it). A pending fold of more copies is applied
// first (host challenges only) on a table of all wires; linear frames take copy 0
// after the pending fold from the bytes at once. out: [0] frames on tables, [1]
// linear ones; `forms` (if any) come before them.
constexpr int kFinishKinds = 2;

bool plan_finish_frame(Batch* B, Frame* f, fp2* d_wires, fp2* d_beta, RoundLaunch (&out)[kFinishKinds])
{
    if (f->pending && !f->linear && f->n_phys > 2 &&
        (device_fold_blocked(f) || !apply_fold(f, B->stream, &B->launches)))
        return false;
    Job j = base_job(f);
    j.kind = f->pending ? 1 : 0;  // a pending fold of the last two copies
    j.fin = d_wires ? d_wires : f->fin;
    j.fin_beta = d_beta ? d_beta : f->fin + f->n_wires;
    RoundLaunch& L = out[f->linear ? 1 : 0];
    L.kind = 8;
    j.tiles = j.groups = 1;
    L.max_w = std::max(L.max_w, f->n_wires);
    L.jobs.push_back(j);
    L.rdev.push_back(f->pending ? f->r_dev : nullptr);
    return true;
}

bool plan_finish(Batch* B, fp2* const* d_wires, fp2* const* d_beta, std::vector<RoundLaunch>& forms,
                 RoundLaunch (&out)[kFinishKinds])
{
    Ctx* c = ctx();
    if (!c) return false;
    std::vector<Frame*> fresh;
    for (size_t i = 0; i < B->frames.size(); ++i) {
        Frame* f = B->frames[i];
        if (!f->configured) continue;
        if (!f->loaded) {
            set_error(TP_ERR_ARG, "frame %zu has no table", i);
            return false;
        }
        if (f->linear && !f->forms_done) fresh.push_back(f);   // their bytes are copied by the forms
        if (!plan_finish_frame(B, f, d_wires ? d_wires[i] : nullptr, d_beta ? d_beta[i] : nullptr, out)) return false;
    }
    plan_linear_finish(out[1].jobs);
    plan_forms(fresh, forms, c->n_sm);
    return true;
}

bool launch_finish_kind(const Job* d_jobs, const RoundLaunch& L, int which, cudaStream_t s, int* launches)
{
    return which == 0 ? launch_finish(d_jobs, (int)L.jobs.size(), L.max_w, s, launches)
                      : launch_linear_finish(d_jobs, L.jobs, s, launches);
}

bool launch_finishes(Batch* B, std::vector<RoundLaunch>& forms, RoundLaunch (&fin)[kFinishKinds])
{
    for (RoundLaunch& L : forms)
        if (!launch_planned(B, L)) return false;
    for (int q = 0; q < kFinishKinds; ++q) {
        RoundLaunch& L = fin[q];
        if (L.jobs.empty()) continue;
        if (!ensure_workspace(B, L.jobs.size(), 1)) return false;
        set_workspace_ptrs(B, L.jobs);
        if (!upload_jobs(B, L.jobs.data(), L.jobs.size(), L.rdev)) return false;
        if (!launch_finish_kind(B->d_jobs, L, q, B->stream, &B->launches)) return false;
    }
    return true;
}

}  // namespace

bool batch_finish(Batch* B, fp2* const* d_wires, fp2* const* d_beta)
{
    std::vector<RoundLaunch> forms;
    RoundLaunch fin[kFinishKinds];
    return plan_finish(B, d_wires, d_beta, forms, fin) && launch_finishes(B, forms, fin);
}

namespace {

struct GraphOp {
    int type = 0;          // 0 round launch, 1 VOLE round, 2 finish, 3 all rounds left in one launch
    int fin = 0;           // 2: which of the finish kinds
    RoundLaunch L;
    size_t job_off = 0, patch_off = 0, n_patch = 0;
    int round = 0;
};

template <class T>
bool grow_dev(T*& p, size_t& cap, size_t n, cudaStream_t s)
{
    if (n <= cap) return true;
    dev_free(p, s);
    cap = std::max(n, cap * 2);
    p = static_cast<T*>(dev_alloc(sizeof(T) * cap, s));
    if (!p) cap = 0;
    return p != nullptr;
}

}  // namespace

bool batch_vole_rounds_graph(Batch* B, u64* d_claims, void* d_states, void* d_vole_states, const fp2* d_u,
                             const fp2* d_v, long long count, int layer, fp2* d_chal, fp2* d_proof,
                             fp2* const* d_wires, fp2* const* d_beta)
{
    Ctx* c = ctx();
    if (!c) return false;
    cudaStream_t s = B->stream;
    if (!s) {
        set_error(TP_ERR_ARG, "the graph path needs a stream of the caller's (the legacy stream cannot capture)");
        return false;
    }
    const int nB = (int)B->frames.size();
    // rounds per frame; frames of different sizes (uneven batches) leave the
    // round loop after their own last round: their VOLE round is skipped (the
    // frame's entry in a device array of rounds) and they get no more claims
    int rounds = 0;
    bool uneven = false;
    std::vector<int> fr_rounds((size_t)nB);
    for (int i = 0; i < nB; ++i) {
        Frame* f = B->frames[(size_t)i];
        if (!f->configured || f->n_copies < 2) {
            set_error(TP_ERR_ARG, "every frame of the batch needs at least one round");
            return false;
        }
        int r = 0;
        while ((2 << r) <= f->n_copies) ++r;
        fr_rounds[(size_t)i] = r;
        if (i && r != rounds) uneven = true;
        rounds = std::max(rounds, r);
    }
    // ---- plan every launch (advances the frames as the launches will)
    std::vector<GraphOp> ops;
    std::vector<u64*> claim_ptrs((size_t)nB);
    auto push = [&](RoundLaunch& L, int type) {
        GraphOp op;
        op.type = type;
        op.L = std::move(L);
        ops.push_back(std::move(op));
    };
    int k = 0;
    for (; k < rounds; ++k) {
        // once only frames on vectors have rounds left, and few pairs, each runs the rest
        // of its rounds, transcript included, in one CTA
        bool fuse = true;
        for (const Frame* f : B->frames)
            fuse = fuse && f->loaded && (f->n_copies < 2 || (f->linear && few_left(f)));
        if (fuse) break;
        for (int i = 0; i < nB; ++i) claim_ptrs[(size_t)i] = d_claims + 8 * ((size_t)nB * k + i);
        std::vector<RoundLaunch> plan;
        if (!plan_claims(B, claim_ptrs.data(), plan)) return false;
        for (RoundLaunch& L : plan) push(L, 0);
        GraphOp v;
        v.type = 1;
        v.round = k;
        ops.push_back(v);
        for (int i = 0; i < nB; ++i)
            if (k < fr_rounds[(size_t)i] && !batch_fold_dev(B, i, d_chal + (size_t)nB * k + i)) return false;
    }
    if (k < rounds) {
        std::vector<RoundLaunch> plan;
        plan_forms(B->frames, plan, c->n_sm);
        for (RoundLaunch& L : plan) push(L, 0);
        RoundLaunch L;
        for (int i = 0; i < nB; ++i) {
            Frame* f = B->frames[(size_t)i];
            const int left = fr_rounds[(size_t)i] - k;
            if (left <= 0) continue;
            RoundLaunch one;
            plan_given(f, left, d_claims + 8 * ((size_t)nB * k + i), f2zero(), one);
            one.jobs[0].frame = i;
            f->r_dev = d_chal + (size_t)nB * (fr_rounds[(size_t)i] - 1) + i;   // the last fold's challenge
            L.kind = one.kind;
            L.jobs.push_back(one.jobs[0]);
            L.rdev.push_back(one.rdev[0]);
        }
        push(L, 3);
        ops.back().round = k;
    }
    {
        std::vector<RoundLaunch> forms;
        RoundLaunch fin[kFinishKinds];
        if (!plan_finish(B, d_wires, d_beta, forms, fin)) return false;
        for (RoundLaunch& L : forms) push(L, 0);
        for (int q = 0; q < kFinishKinds; ++q)
            if (!fin[q].jobs.empty()) {
                push(fin[q], 2);
                ops.back().fin = q;
            }
    }
    // ---- workspace, one job table and one patch table
    size_t max_jobs = 1, max_ctas = 1, n_jobs = 0, n_patch = 0;
    for (GraphOp& op : ops) {
        if (op.type == 1) continue;
        max_jobs = std::max(max_jobs, op.L.jobs.size());
        if (op.type == 0) max_ctas = std::max(max_ctas, launch_ctas(op.L.jobs));
    }
    if (!ensure_workspace(B, max_jobs, max_ctas)) return false;
    for (GraphOp& op : ops) {
        if (op.type == 1) continue;
        if (op.type != 3) set_workspace_ptrs(B, op.L.jobs);
        op.job_off = n_jobs;
        op.patch_off = n_patch;
        for (const fp2* r : op.L.rdev) op.n_patch += r ? 1 : 0;
        n_jobs += op.L.jobs.size();
        n_patch += op.n_patch;
    }
    struct Patch {
        const fp2* r;
        long long job;
    };
    static_assert(sizeof(Patch) == 16, "patch layout (patch_r_kernel's RPatch)");
    // the patch table, then (uneven batches) the rounds of each frame
    const size_t bytes_jobs = sizeof(Job) * n_jobs, bytes_patch_only = sizeof(Patch) * std::max<size_t>(1, n_patch);
    const size_t bytes_patch = bytes_patch_only + (uneven ? sizeof(int) * (size_t)nB : 0);
    if (!grow_dev(B->d_table, B->cap_table, n_jobs, s)) return false;
    {
        unsigned char* pt = static_cast<unsigned char*>(B->d_ptable);
        size_t cap = B->cap_ptable;
        if (!grow_dev(pt, cap, bytes_patch, s)) return false;
        B->d_ptable = pt;
        B->cap_ptable = cap;
    }
    if (!B->staged) TP_CUDA_OK(cudaEventCreateWithFlags(&B->staged, cudaEventDisableTiming), "stage event");
    TP_CUDA_OK(cudaEventSynchronize(B->staged), "stage reuse");   // the previous upload has read the stage
    if (bytes_jobs + bytes_patch > B->cap_stage) {
        if (B->h_stage) cudaFreeHost(B->h_stage);
        B->cap_stage = std::max(bytes_jobs + bytes_patch, 2 * B->cap_stage);
        if (cuda_failed(cudaMallocHost(&B->h_stage, B->cap_stage), "pinned stage")) {
            B->h_stage = nullptr;
            B->cap_stage = 0;
            return false;
        }
    }
    Job* hj = static_cast<Job*>(B->h_stage);
    Patch* hp = reinterpret_cast<Patch*>(static_cast<unsigned char*>(B->h_stage) + bytes_jobs);
    for (const GraphOp& op : ops) {
        if (op.type == 1) continue;
        std::memcpy(hj + op.job_off, op.L.jobs.data(), sizeof(Job) * op.L.jobs.size());
        size_t q = op.patch_off;
        for (size_t j = 0; j < op.L.rdev.size(); ++j)
            if (op.L.rdev[j]) hp[q++] = Patch{op.L.rdev[j], (long long)(op.job_off + j)};
    }
    int* d_rounds = nullptr;
    if (uneven) {
        std::memcpy(reinterpret_cast<unsigned char*>(hp) + bytes_patch_only, fr_rounds.data(), sizeof(int) * (size_t)nB);
        d_rounds = reinterpret_cast<int*>(static_cast<unsigned char*>(B->d_ptable) + bytes_patch_only);
    }
    TP_CUDA_OK(cudaMemcpyAsync(B->d_table, hj, bytes_jobs, cudaMemcpyHostToDevice, s), "job table");
    if (n_patch || uneven)
        TP_CUDA_OK(cudaMemcpyAsync(B->d_ptable, hp, bytes_patch, cudaMemcpyHostToDevice, s), "patch table");
    TP_CUDA_OK(cudaEventRecord(B->staged, s), "stage event");
    // ---- the graph: captured once per shape, replayed after
    std::vector<long long> key = {(long long)(size_t)s, (long long)(size_t)B->d_table, (long long)(size_t)B->d_ptable,
                                  (long long)(size_t)d_states, (long long)(size_t)d_vole_states,
                                  (long long)(size_t)d_u, (long long)(size_t)d_v, count, layer,
                                  (long long)(size_t)d_chal, (long long)(size_t)d_proof, (long long)nB,
                                  (long long)uneven, (long long)(size_t)d_claims};
    int kernels = 0;
    for (const GraphOp& op : ops) {
        key.push_back(op.type);
        key.push_back(op.L.kind);
        key.push_back((long long)op.job_off);
        key.push_back((long long)op.L.jobs.size());
        key.push_back((long long)op.patch_off);
        key.push_back((long long)op.n_patch);
        key.push_back(op.L.max_w);
        key.push_back(op.fin);
        key.push_back(op.round);
        for (const Job& j : op.L.jobs) {
            key.push_back(j.tiles);
            key.push_back(j.groups);
            key.push_back(j.wpg);
            key.push_back(j.pw);
            key.push_back(j.stride);
            key.push_back(j.chunks);
            key.push_back(j.W);
            key.push_back(j.nf + j.has_r);
        }
        kernels += (op.type == 1) ? 1 : 1 + (op.n_patch ? 1 : 0);
    }
    if (!B->graph || key != B->graph_key) {
        if (B->graph) {
            cudaGraphExecDestroy(B->graph);
            B->graph = nullptr;
        }
        if (!prepare_round_kernels() || !prepare_linear_kernels()) return false;
        TP_CUDA_OK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "begin capture");
        bool ok = true;
        int dummy = 0;
        for (const GraphOp& op : ops) {
            if (!ok) break;
            if (op.type == 1) {
                char label[40];
                std::snprintf(label, sizeof(label), "sc-%d-%d", layer, op.round);
                ok = launch_vole_round_batch(d_states, d_vole_states, nB, d_claims + 8 * (size_t)nB * op.round,
                                             d_u, d_v, count, label, d_chal + (size_t)nB * op.round,
                                             d_proof ? d_proof + 5 * (size_t)nB * op.round : nullptr, s, d_rounds,
                                             op.round);
                continue;
            }
            if (op.n_patch) {
                patch_r_kernel<<<(unsigned)((op.n_patch + 127) / 128), 128, 0, s>>>(
                    B->d_table, static_cast<const RPatch*>(B->d_ptable) + op.patch_off, (int)op.n_patch);
                ok = !cuda_failed(cudaGetLastError(), "challenge patch");
            }
            if (!ok) break;
            if (op.type == 0) {
                ok = launch_any(B->d_table + op.job_off, op.L, s, &dummy);
            } else if (op.type == 3) {
                const VoleRounds v = {d_states, d_vole_states, d_u, d_v, d_chal, d_proof, count, nB, layer};
                ok = launch_linear_rounds(B->d_table + op.job_off, (int)op.L.jobs.size(), &v, op.round,
                                          8 * (long long)nB, s, &dummy);
            } else {
                ok = launch_finish_kind(B->d_table + op.job_off, op.L, op.fin, s, &dummy);
            }
        }
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(s, &g);
        if (!ok || cuda_failed(e, "end capture")) {
            if (g) cudaGraphDestroy(g);
            return false;
        }
        const cudaError_t ie = cudaGraphInstantiate(&B->graph, g, 0);
        cudaGraphDestroy(g);
        if (cuda_failed(ie, "graph instantiate")) {
            B->graph = nullptr;
            return false;
        }
        B->graph_key = key;
        B->graph_kernels = kernels;
    }
    TP_CUDA_OK(cudaGraphLaunch(B->graph, s), "graph launch");
    B->launches += B->graph_kernels;
    ++B->graph_replays;
    return true;
}

void batch_tune_enable(bool on) { g_tune_on = on; }

int batch_tune_table(int* kind, int* bucket, int* ctas_per_sm, int max)
{
    Ctx* c = ctx();
    std::lock_guard<std::mutex> lk(tune_mutex());
    int n = 0;
    for (const auto& kv : tune_table()) {
        if (c && kv.first.device != c->device) continue;
        if (n < max) {
            kind[n] = kv.first.kind;
            bucket[n] = kv.first.bucket;
            ctas_per_sm[n] = kv.second;
        }
        ++n;
    }
    return n;
}

bool batch_tune_set(int kind, int bucket, int ctas_per_sm)
{
    Ctx* c = ctx();
    if (!c) return false;
    if (kind < 0 || kind > 3 || bucket < 0 || bucket > 62 || ctas_per_sm < 1 || ctas_per_sm > 64) {
        set_error(TP_ERR_ARG, "tune entry (%d, %d, %d) out of range", kind, bucket, ctas_per_sm);
        return false;
    }
    std::lock_guard<std::mutex> lk(tune_mutex());
    tune_table()[TuneKey{c->device, kind, bucket}] = ctas_per_sm;
    return true;
}

bool batch_finish_frame(Batch* B, int i, fp2* d_wires, fp2* d_beta)
{
    if (i < 0 || i >= (int)B->frames.size()) {
        set_error(TP_ERR_ARG, "frame index %d outside the batch", i);
        return false;
    }
    Frame* f = B->frames[(size_t)i];
    if (!f->configured || !f->loaded) {
        set_error(TP_ERR_ARG, "frame %d is not configured", i);
        return false;
    }
    Ctx* c = ctx();
    if (!c) return false;
    std::vector<RoundLaunch> forms;
    RoundLaunch fin[kFinishKinds];
    const bool fresh = f->linear && !f->forms_done;
    if (!plan_finish_frame(B, f, d_wires, d_beta, fin)) return false;
    plan_linear_finish(fin[1].jobs);
    if (fresh) plan_forms({f}, forms, c->n_sm);
    if (!launch_finishes(B, forms, fin)) return false;
    batch_release(B, i, false);
    return true;
}

void batch_release(Batch* B, int i, bool free_buffers)
{
    if (i < 0 || i >= (int)B->frames.size()) return;
    Frame* f = B->frames[(size_t)i];
    f->configured = f->loaded = false;
    f->n_copies = 0;
    f->pending = false;
    f->r_dev = nullptr;
    if (free_buffers) {
        cudaStream_t s = B->stream;
        if (!f->borrowed0) dev_free(f->buf[0], s);
        dev_free(f->buf[1], s);
        dev_free(f->beta[0], s);
        dev_free(f->beta[1], s);
        f->buf[0] = f->buf[1] = f->beta[0] = f->beta[1] = nullptr;
        f->cap0 = f->cap1 = f->capb = 0;
        f->borrowed0 = false;
        linear_free(f, s);
    }
}

void batch_reset(Batch* B)
{
    for (Frame* f : B->frames) {
        f->configured = f->loaded = false;
        f->n_copies = 0;
    }
}

void batch_destroy(Batch* B)
{
    if (!B) return;
    cudaStream_t s = B->stream;
    for (Frame* f : B->frames) {
        if (!f->borrowed0) dev_free(f->buf[0], s);
        dev_free(f->buf[1], s);
        dev_free(f->beta[0], s);
        dev_free(f->beta[1], s);
        dev_free(f->fin, s);
        dev_free(f->out8, s);
        linear_free(f, s);
        dev_free(f->rs, s);
        free_gate_form(f->form, s);
        delete f;
    }
    dev_free(B->forms, s);
    dev_free(B->d_jobs, s);
    dev_free(B->partials, s);
    dev_free(B->tickets, s);
    dev_free(B->d_patch, s);
    dev_free(B->d_table, s);
    dev_free(B->d_ptable, s);
    if (B->graph) cudaGraphExecDestroy(B->graph);
    if (B->staged) {
        cudaEventSynchronize(B->staged);
        cudaEventDestroy(B->staged);
    }
    if (B->h_stage) cudaFreeHost(B->h_stage);
    delete B;
}

Batch* session_create(int n_gates, const int* type, const int* in0, const int* in1,
                      const u64* z_re, const u64* z_im, int n_copies, int n_wires, cudaStream_t s)
{
    Batch* B = batch_create(1, s);
    if (!B) return nullptr;
    if (!batch_set_gates(B, 0, n_gates, type, in0, in1, z_re, z_im, n_copies, n_wires)) {
        batch_destroy(B);
        return nullptr;
    }
    return B;
}

bool session_claim(Batch* B, u64 out8[8])
{
    if (!batch_claim(B, nullptr)) return false;
    TP_CUDA_OK(cudaMemcpyAsync(out8, B->frames[0]->out8, 64, cudaMemcpyDeviceToHost, B->stream),
               "D2H claim");
    TP_CUDA_OK(cudaStreamSynchronize(B->stream), "claim");
    return true;
}

bool session_finish(Batch* B, u64* w_re, u64* w_im, u64* b_re, u64* b_im)
{
    if (!batch_finish(B, nullptr, nullptr)) return false;
    Frame* f = B->frames[0];
    std::vector<fp2> h((size_t)f->n_wires + 1);
    TP_CUDA_OK(cudaMemcpyAsync(h.data(), f->fin, sizeof(fp2) * h.size(), cudaMemcpyDeviceToHost,
                               B->stream), "D2H finish");
    TP_CUDA_OK(cudaStreamSynchronize(B->stream), "finish");
    for (int w = 0; w < f->n_wires; ++w) {
        w_re[w] = h[w].re;
        w_im[w] = h[w].im;
    }
    *b_re = h[f->n_wires].re;
    *b_im = h[f->n_wires].im;
    return true;
}

}  // namespace tp
