// The learned preconditioner's network: a 3-level 3-D convolutional U-Net
// (channels c1/c2/c3, 3x3x3 kernels, BF16 weights and activations, FP32
// accumulation), trained and run by the project's own kernels
// (pps_unet_conv.cu).  No reference counterpart.
//
//   x0 --conv0,relu--> e1a --conv1,relu--> e1 ----------------------------(skip)--+
//                                           |pool                                 |
//             p1 --conv2,relu--> e2a --conv3,relu--> e2 -------------(skip)--+     |
//                                                     |pool                  |     |
//                        p2 --conv4,relu--> e3a --conv5,relu--> e3 --up--> [e3|e2] |
//                                                       conv6,relu -> d2a -> conv7,relu -> d2
//                                                                          --up--> [d2|e1]
//                                                       conv8,relu -> d1a -> conv9,relu -> d1
//                                                       conv10 (linear, 1 channel) -> out
//
// Input and output are one channel; the input is scaled to unit RMS and the output
// scaled back by the same factor, so the map is positively homogeneous like A^-1.
#include "../../include/pps.h"
#include "pps_unet_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <random>
#include <string>
#include <vector>

using namespace pps;
using namespace pps::unet;

namespace {

struct UFail {};

#define UK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) {                                                              \
            pps_internal_set_error((std::string(#call) + ": " + cudaGetErrorString(e_)).c_str()); \
            throw UFail{};                                                                    \
        }                                                                                     \
    } while (0)

struct Layer {
    int cin, cout;         // real channels
    int cin_p, cout_p;     // padded to multiples of 16
    bool relu;
    size_t w, b;           // offsets of W [27][cin_p][cout_p] and b [cout_p] in the padded arrays
    size_t rw, rb;         // offsets in the real (unpadded) flat parameter vector
};

int pad16(int c) { return (c + 15) / 16 * 16; }

struct Acts {
    Dims s1{0, 0, 0}, s2{0, 0, 0}, s3{0, 0, 0};   // grid of each level
    bf16 *e1a = nullptr, *e1 = nullptr, *d1a = nullptr, *d1 = nullptr;
    bf16 *e2a = nullptr, *e2 = nullptr, *d2a = nullptr, *d2 = nullptr;
    bf16 *e3a = nullptr, *e3 = nullptr, *p1 = nullptr, *p2 = nullptr;   // p: pooled e1, e2
    // gradients: of the outputs of layers 9, 8, 7, 6, 5, 4, 2, 0 (masked where stored), of
    // the two concatenations and the two pooled tensors, and of the dense output
    bf16 *g_d1 = nullptr, *g_d1a = nullptr, *g_cat1 = nullptr, *g_d2a = nullptr, *g_cat2 = nullptr, *g_e3a = nullptr,
         *g_p2 = nullptr, *g_e2a = nullptr, *g_p1 = nullptr, *g_e1a = nullptr, *g_d2 = nullptr, *g_e3 = nullptr;
    float* g_out = nullptr;
    bool grads = false;
};

}  // namespace

struct pps_unet {
    int c1, c2, c3;
    int linear = 0;        // 1: identity activations (a learned linear multigrid-like operator)
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<Layer> L;
    size_t npad = 0, nreal = 0;
    float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;   // FP32 master, grads, Adam moments
    bf16 *WP = nullptr, *WB = nullptr;   // BF16 weights in fragment order: forward, data gradient
    PackTable pt{};
    float* dtmp = nullptr; // device scalars: rms of the input, rms of the gradient
    double* dloss = nullptr;   // behind the gradients in one allocation: one fill zeroes both
    RmsScratch* drms = nullptr;
    int step = 0;
    Acts A;
    unsigned long long version = 0;   // of what a captured forward pass holds: A's buffers, the activation
    // Page-locked landing place of parameters and gradients (+ the loss behind them),
    // allocated when first read; reads of one network from several threads take turns.
    mutable float* stage = nullptr;
    mutable std::mutex stage_lock;
};

namespace {

void free_acts(Acts& A)
{
    bf16* b[] = {A.e1a, A.e1, A.d1a, A.d1, A.e2a, A.e2, A.d2a, A.d2, A.e3a, A.e3, A.p1, A.p2, A.g_d1, A.g_d1a, A.g_cat1, A.g_d2a,
                 A.g_cat2, A.g_e3a, A.g_p2, A.g_e2a, A.g_p1, A.g_e1a, A.g_d2, A.g_e3};
    for (bf16* q : b)
        if (q) cudaFree(q);
    if (A.g_out) cudaFree(A.g_out);
    A = Acts();
}

bf16* balloc(long long n)
{
    bf16* p = nullptr;
    UK(cudaMalloc((void**)&p, sizeof(bf16) * (size_t)n));
    return p;
}

void ensure_acts(pps_unet* u, int nx, int ny, int nz, bool grads)
{
    Acts& A = u->A;
    if (A.s1.W == nx && A.s1.H == ny && A.s1.D == nz && (A.grads || !grads)) return;
    u->version++;
    free_acts(A);
    const long long v1 = (long long)nx * ny * nz, v2 = v1 / 8, v3 = v2 / 8;
    const int c1 = u->c1, c2 = u->c2, c3 = u->c3;
    A.e1a = balloc(v1 * c1);
    A.e1 = balloc(v1 * c1);
    A.d1a = balloc(v1 * c1);
    A.d1 = balloc(v1 * c1);
    A.e2a = balloc(v2 * c2);
    A.e2 = balloc(v2 * c2);
    A.d2a = balloc(v2 * c2);
    A.d2 = balloc(v2 * c2);
    A.e3a = balloc(v3 * c3);
    A.e3 = balloc(v3 * c3);
    A.p1 = balloc(v2 * c1);
    A.p2 = balloc(v3 * c2);
    if (grads) {
        UK(cudaMalloc((void**)&A.g_out, sizeof(float) * (size_t)v1));
        A.g_d1 = balloc(v1 * c1);
        A.g_d1a = balloc(v1 * c1);
        A.g_cat1 = balloc(v1 * (c2 + c1));
        A.g_d2a = balloc(v2 * c2);
        A.g_cat2 = balloc(v2 * (c3 + c2));
        A.g_e3a = balloc(v3 * c3);
        A.g_p2 = balloc(v3 * c2);
        A.g_e2a = balloc(v2 * c2);
        A.g_p1 = balloc(v2 * c1);
        A.g_e1a = balloc(v1 * c1);
        A.g_d2 = balloc(v2 * c2);
        A.g_e3 = balloc(v3 * c3);
        A.grads = true;
    }
    // the extents last: an allocation that failed half way leaves none
    A.s1 = Dims{nz, ny, nx};
    A.s2 = Dims{nz / 2, ny / 2, nx / 2};
    A.s3 = Dims{nz / 4, ny / 4, nx / 4};
}

const float* Bf(const pps_unet* u, int l) { return u->P + u->L[(size_t)l].b; }

Src plain(const bf16* X, int ld, int c0 = 0)
{
    Src s;
    s.X = X;
    s.ld = ld;
    s.c0 = c0;
    return s;
}
// the concatenation [upsampled coarse tensor | skip tensor]
Src concat(const bf16* up, int c_up, const bf16* skip, int c_skip)
{
    Src s = plain(skip, c_skip, -c_up);
    s.kind = SRC_UP;
    s.up = up;
    s.ld_up = c_up;
    s.c_up = c_up;
    return s;
}
Src dense(const float* in, const float* rms_dev)
{
    Src s;
    s.kind = SRC_DENSE;
    s.dense = in;
    s.rms = rms_dev;
    return s;
}
// the gradient of a skip tensor: its slot of the concatenation's gradient plus the pooled path
Src skip(const bf16* gcat, int ld, int c0, const bf16* gpool, int c, const bf16* mask)
{
    Src s = plain(gcat, ld, c0);
    s.kind = SRC_SKIP;
    s.up = gpool;
    s.ld_up = c;
    s.mask = mask;
    s.ldm = c;
    return s;
}

// What each layer reads; with `rms_dev` the input is scaled by 1/(*rms_dev).
Src layer_input(const pps_unet* u, int l, const float* in, const float* rms_dev)
{
    const Acts& A = u->A;
    const int c1 = u->c1, c2 = u->c2, c3 = u->c3;
    switch (l) {
    case 0: return dense(in, rms_dev);
    case 1: return plain(A.e1a, c1);
    case 2: return plain(A.p1, c1);
    case 3: return plain(A.e2a, c2);
    case 4: return plain(A.p2, c2);
    case 5: return plain(A.e3a, c3);
    case 6: return concat(A.e3, c3, A.e2, c2);
    case 7: return plain(A.d2a, c2);
    case 8: return concat(A.d2, c2, A.e1, c1);
    case 9: return plain(A.d1a, c1);
    default: return plain(A.d1, c1);
    }
}

const Dims& layer_dims(const pps_unet* u, int l)
{
    return l == 4 || l == 5 ? u->A.s3 : (l == 2 || l == 3 || l == 6 || l == 7) ? u->A.s2 : u->A.s1;
}

// The forward pass: every layer one convolution, upsampling and concatenations folded
// into its loads, and the two poolings.  `last` is what the last layer does with its
// sums: the dense output, or the loss and its gradient.
void forward(pps_unet* u, const float* in, const float* rms_dev, Epi last)
{
    Acts& A = u->A;
    bf16* out[10] = {A.e1a, A.e1, A.e2a, A.e2, A.e3a, A.e3, A.d2a, A.d2, A.d1a, A.d1};
    for (int l = 0; l < UNET_LAYERS; l++) {
        const Layer& L = u->L[(size_t)l];
        Epi e = last;
        if (l < 10) {
            e = Epi();
            e.Y = out[l];
            e.ld = L.cout_p;
            e.relu = u->linear ? 0 : 1;
        }
        e.bias = Bf(u, l);
        if (l == 2) gather8(A.s2, A.e1, u->c1, u->c1, 0.125f, nullptr, A.p1, u->stream);
        if (l == 4) gather8(A.s3, A.e2, u->c2, u->c2, 0.125f, nullptr, A.p2, u->stream);
        conv(layer_dims(u, l), layer_input(u, l, in, rms_dev), u->WP + L.w, L.cin_p, L.cout_p, e, u->stream);
    }
}

// Gradients of the parameters from A.g_out, the gradient of the dense output: the data
// gradients layer by layer (each a convolution of the output gradient G_l with the
// mirrored weights), then all weight and bias gradients in one launch.
void backward(pps_unet* u, const float* in)
{
    Acts& A = u->A;
    const int c1 = u->c1, c2 = u->c2, c3 = u->c3;
    const bool R = !u->linear;
    const Src G[UNET_LAYERS] = {
        plain(A.g_e1a, c1),
        skip(A.g_cat1, c2 + c1, c2, A.g_p1, c1, R ? A.e1 : nullptr),
        plain(A.g_e2a, c2),
        skip(A.g_cat2, c3 + c2, c3, A.g_p2, c2, R ? A.e2 : nullptr),
        plain(A.g_e3a, c3),
        plain(A.g_e3, c3),
        plain(A.g_d2a, c2),
        plain(A.g_d2, c2),
        plain(A.g_d1a, c1),
        plain(A.g_d1, c1),
        dense(A.g_out, nullptr),
    };
    // gradient of layer l's input, and the activation whose ReLU it passes (where that
    // input is one layer's stored output)
    bf16* gin[UNET_LAYERS] = {nullptr, A.g_e1a, A.g_p1, A.g_e2a, A.g_p2, A.g_e3a, A.g_cat2, A.g_d2a, A.g_cat1, A.g_d1a, A.g_d1};
    const bf16* act[UNET_LAYERS] = {nullptr, A.e1a, nullptr, A.e2a, nullptr, A.e3a, nullptr, A.d2a, nullptr, A.d1a, A.d1};
    for (int l = 10; l >= 1; l--) {
        const Layer& L = u->L[(size_t)l];
        Epi e;
        e.Y = gin[l];
        e.ld = L.cin_p;
        e.mask = R ? act[l] : nullptr;
        e.ldm = L.cin_p;
        // gradients of the upsampled tensors: their channels lie first in the concatenation's
        if (l == 7) gather8(A.s2, A.g_cat1, c2 + c1, c2, 1.0f, R ? A.d2 : nullptr, A.g_d2, u->stream);
        if (l == 5) gather8(A.s3, A.g_cat2, c3 + c2, c3, 1.0f, R ? A.e3 : nullptr, A.g_e3, u->stream);
        conv(layer_dims(u, l), G[l], u->WB + L.w, L.cout_p, L.cin_p, e, u->stream);
    }
    WgTable T;
    T.n = UNET_LAYERS;
    for (int l = 0; l < UNET_LAYERS; l++) {
        const Layer& L = u->L[(size_t)l];
        WgLayer& W = T.L[l];
        W.d = layer_dims(u, l);
        W.X = layer_input(u, l, in, nullptr);
        W.G = G[l];
        W.Cin = L.cin_p;
        W.Cout = L.cout_p;
        W.dW = u->G + L.w;
        W.db = u->G + L.b;
    }
    wgrad(T, u->stream);
}

pps_status check_dims(int nx, int ny, int nz)
{
    if (nx < 4 || ny < 4 || nz < 4 || nx % 4 || ny % 4 || nz % 4) {
        pps_internal_set_error("the U-Net needs every extent to be a multiple of 4 (two 2x poolings)");
        return PPS_ERR_INVALID_ARG;
    }
    return PPS_OK;
}

template <typename Fn>
pps_status uguard(Fn&& fn)
{
    const unsigned long long f0 = pps::launch_failures();
    try {
        const pps_status rc = fn();
        return rc >= 0 && pps::launch_failures() != f0 ? PPS_ERR_CUDA : rc;
    } catch (const UFail&) {
        return PPS_ERR_CUDA;
    } catch (const std::bad_alloc&) {
        pps_internal_set_error("host allocation failed");
        return PPS_ERR_OUT_OF_MEMORY;
    }
}

}  // namespace

// internal: run the forward pass on the U-Net's stream-independent buffers (used
// by the solver's learned preconditioner).  in/out dense [nz][ny][nx] FP32.
pps_status pps_internal_unet_apply(pps_unet* u, int nx, int ny, int nz, const float* in, float* out, float gain,
                                   cudaStream_t s)
{
    if (check_dims(nx, ny, nz) != PPS_OK) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        struct OnStream {   // the network's own stream again afterwards, an error included
            pps_unet* u;
            cudaStream_t own;
            ~OnStream() { u->stream = own; }
        } on{u, u->stream};
        u->stream = s;
        ensure_acts(u, nx, ny, nz, false);
        const long long nv = (long long)nx * ny * nz;
        rms(nv, in, u->dtmp, u->drms, s);
        Epi last;
        last.dense_out = out;
        last.rms = u->dtmp;
        last.gain = gain;
        forward(u, in, u->dtmp, last);
        return PPS_OK;
    });
}

unsigned long long pps_internal_unet_version(const pps_unet* u) { return u->version; }

extern "C" {

pps_status pps_unet_create(int c1, int c2, int c3, unsigned long long seed, int device, pps_unet** out)
{
    if (!out || c1 < 16 || c2 < 16 || c3 < 16 || c1 % 16 || c2 % 16 || c3 % 16 || c3 + c2 > 96 || c2 + c1 > 96) {
        pps_internal_set_error("U-Net channels must be multiples of 16 with c3+c2 <= 96");
        return PPS_ERR_INVALID_ARG;
    }
    *out = nullptr;
    pps_unet* u = new (std::nothrow) pps_unet();
    if (!u) return PPS_ERR_OUT_OF_MEMORY;
    u->c1 = c1;
    u->c2 = c2;
    u->c3 = c3;
    const int spec[11][3] = {{1, c1, 1},  {c1, c1, 1}, {c1, c2, 1}, {c2, c2, 1},      {c2, c3, 1}, {c3, c3, 1},
                             {c3 + c2, c2, 1}, {c2, c2, 1}, {c2 + c1, c1, 1}, {c1, c1, 1}, {c1, 1, 0}};
    size_t off = 0, roff = 0;
    for (auto& sp : spec) {
        Layer l;
        l.cin = sp[0];
        l.cout = sp[1];
        l.relu = sp[2] != 0;
        l.cin_p = pad16(l.cin);
        l.cout_p = pad16(l.cout);
        l.w = off;
        off += (size_t)27 * l.cin_p * l.cout_p;
        l.b = off;
        off += (size_t)l.cout_p;
        l.rw = roff;
        roff += (size_t)27 * l.cin * l.cout;
        l.rb = roff;
        roff += (size_t)l.cout;
        u->L.push_back(l);
    }
    u->npad = off;
    u->nreal = roff;
    pps_status rc = uguard([&]() -> pps_status {
        UK(cudaSetDevice(device));
        u->device = device;
        UK(cudaStreamCreateWithFlags(&u->stream, cudaStreamNonBlocking));
        UK(conv_prepare());
        // each layer's parameters are a multiple of 16 floats, so the loss behind the
        // gradients is 8-byte aligned
        float** f[] = {&u->P, &u->G, &u->M, &u->V};
        for (float** q : f) {
            UK(cudaMalloc((void**)q, sizeof(float) * u->npad + sizeof(double)));
            UK(cudaMemsetAsync(*q, 0, sizeof(float) * u->npad + sizeof(double), u->stream));
        }
        u->dloss = reinterpret_cast<double*>(u->G + u->npad);
        for (bf16** q : {&u->WP, &u->WB}) {
            UK(cudaMalloc((void**)q, sizeof(bf16) * u->npad));
            UK(cudaMemsetAsync(*q, 0, sizeof(bf16) * u->npad, u->stream));
        }
        UK(cudaMalloc((void**)&u->dtmp, sizeof(float) * 4));
        UK(cudaMalloc((void**)&u->drms, sizeof(RmsScratch)));
        UK(cudaMemsetAsync(u->drms, 0, sizeof(RmsScratch), u->stream));
        u->pt.n = UNET_LAYERS;
        for (int l = 0; l < UNET_LAYERS; l++) {
            u->pt.w[l] = (int)u->L[(size_t)l].w;
            u->pt.cin[l] = u->L[(size_t)l].cin_p;
            u->pt.cout[l] = u->L[(size_t)l].cout_p;
        }
        // He initialisation of the real weights, zero biases
        std::vector<float> h(u->npad, 0.0f);
        std::mt19937_64 rng(seed);
        for (const Layer& l : u->L) {
            std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (27.0f * l.cin)));
            for (int t = 0; t < 27; t++)
                for (int ci = 0; ci < l.cin; ci++)
                    for (int co = 0; co < l.cout; co++)
                        h[l.w + ((size_t)t * l.cin_p + ci) * l.cout_p + co] = nd(rng) * (l.relu ? 1.0f : 0.1f);
        }
        UK(cudaMemcpyAsync(u->P, h.data(), sizeof(float) * u->npad, cudaMemcpyHostToDevice, u->stream));
        pack(u->pt, (int)u->npad, u->P, u->WP, u->WB, u->stream);
        UK(cudaStreamSynchronize(u->stream));
        return PPS_OK;
    });
    if (rc != PPS_OK) {
        pps_unet_destroy(u);
        return rc;
    }
    *out = u;
    return PPS_OK;
}

pps_status pps_unet_destroy(pps_unet* u)
{
    if (!u) return PPS_ERR_INVALID_ARG;
    cudaSetDevice(u->device);
    if (u->stream) cudaStreamSynchronize(u->stream);
    free_acts(u->A);
    void* p[] = {u->P, u->G, u->M, u->V, u->WP, u->WB, u->dtmp, u->drms};
    for (void* q : p)
        if (q) cudaFree(q);
    if (u->stage) cudaFreeHost(u->stage);
    if (u->stream) cudaStreamDestroy(u->stream);
    delete u;
    return PPS_OK;
}

int pps_unet_param_count(const pps_unet* u) { return u ? (int)u->nreal : -1; }

pps_status pps_unet_set_activation(pps_unet* u, int linear)
{
    if (!u || (linear != 0 && linear != 1)) return PPS_ERR_INVALID_ARG;
    if (u->linear != linear) u->version++;
    u->linear = linear;
    return PPS_OK;
}

// Flat real-parameter layout: per layer W[27][cin][cout] (tap = kz*9+ky*3+kx) then b[cout].
static void unpad(const pps_unet* u, const float* padded, float* real)
{
    for (const Layer& l : u->L) {
        if (l.cin == l.cin_p && l.cout == l.cout_p) {   // no padding: W and b lie as they are returned
            memcpy(real + l.rw, padded + l.w, sizeof(float) * ((size_t)27 * l.cin * l.cout + l.cout));
            continue;
        }
        for (int t = 0; t < 27; t++)
            for (int ci = 0; ci < l.cin; ci++)
                for (int co = 0; co < l.cout; co++)
                    real[l.rw + ((size_t)t * l.cin + ci) * l.cout + co] = padded[l.w + ((size_t)t * l.cin_p + ci) * l.cout_p + co];
        for (int co = 0; co < l.cout; co++) real[l.rb + co] = padded[l.b + co];
    }
}

// npad floats of `dev` (and the loss behind them, if asked for) read through the
// page-locked stage after the work queued on the network's stream.
static void read_back(const pps_unet* u, const float* dev, float* real, double* loss)
{
    std::lock_guard<std::mutex> hold(u->stage_lock);
    const size_t bytes = sizeof(float) * u->npad + sizeof(double);
    if (!u->stage) UK(cudaHostAlloc((void**)&u->stage, bytes, cudaHostAllocDefault));
    UK(cudaMemcpyAsync(u->stage, dev, bytes, cudaMemcpyDeviceToHost, u->stream));
    UK(cudaStreamSynchronize(u->stream));
    unpad(u, u->stage, real);
    if (loss) memcpy(loss, u->stage + u->npad, sizeof(double));
}

pps_status pps_unet_get_params(const pps_unet* u, float* out)
{
    if (!u || !out) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        UK(cudaSetDevice(u->device));
        read_back(u, u->P, out, nullptr);
        return PPS_OK;
    });
}

pps_status pps_unet_set_params(pps_unet* u, const float* in)
{
    if (!u || !in) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        UK(cudaSetDevice(u->device));
        std::vector<float> h(u->npad, 0.0f);
        for (const Layer& l : u->L) {
            for (int t = 0; t < 27; t++)
                for (int ci = 0; ci < l.cin; ci++)
                    for (int co = 0; co < l.cout; co++)
                        h[l.w + ((size_t)t * l.cin_p + ci) * l.cout_p + co] = in[l.rw + ((size_t)t * l.cin + ci) * l.cout + co];
            for (int co = 0; co < l.cout; co++) h[l.b + co] = in[l.rb + co];
        }
        UK(cudaMemcpyAsync(u->P, h.data(), sizeof(float) * u->npad, cudaMemcpyHostToDevice, u->stream));
        UK(cudaMemsetAsync(u->M, 0, sizeof(float) * u->npad, u->stream));
        UK(cudaMemsetAsync(u->V, 0, sizeof(float) * u->npad, u->stream));
        u->step = 0;
        pack(u->pt, (int)u->npad, u->P, u->WP, u->WB, u->stream);
        UK(cudaStreamSynchronize(u->stream));
        return PPS_OK;
    });
}

pps_status pps_unet_forward(pps_unet* u, int nx, int ny, int nz, const float* in_dev, float* out_dev, int normalize)
{
    if (!u || !in_dev || !out_dev) return PPS_ERR_INVALID_ARG;
    if (check_dims(nx, ny, nz) != PPS_OK) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        UK(cudaSetDevice(u->device));
        ensure_acts(u, nx, ny, nz, false);
        const long long nv = (long long)nx * ny * nz;
        const float* r = nullptr;
        if (normalize) {
            rms(nv, in_dev, u->dtmp, u->drms, u->stream);
            r = u->dtmp;
        }
        Epi last;
        last.dense_out = out_dev;
        last.rms = r;
        forward(u, in_dev, r, last);
        UK(cudaStreamSynchronize(u->stream));
        return PPS_OK;
    });
}

// Queues the loss and the gradients of one sample (u->G, u->dloss behind it).
static void loss_and_grads(pps_unet* u, int nx, int ny, int nz, const float* in, const float* target)
{
    ensure_acts(u, nx, ny, nz, true);
    const long long nv = (long long)nx * ny * nz;
    UK(cudaMemsetAsync(u->G, 0, sizeof(float) * u->npad + sizeof(double), u->stream));   // and the loss
    Epi last;
    last.dense_out = u->A.g_out;
    last.target = target;
    last.loss = u->dloss;
    last.inv_n = (float)(1.0 / (double)nv);
    forward(u, in, nullptr, last);
    backward(u, in);
}

pps_status pps_unet_gradients(pps_unet* u, int nx, int ny, int nz, const float* in_dev, const float* target_dev,
                              float* grads, double* loss)
{
    if (!u || !in_dev || !target_dev || !grads || !loss) return PPS_ERR_INVALID_ARG;
    if (check_dims(nx, ny, nz) != PPS_OK) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        UK(cudaSetDevice(u->device));
        loss_and_grads(u, nx, ny, nz, in_dev, target_dev);
        read_back(u, u->G, grads, loss);
        return PPS_OK;
    });
}

pps_status pps_unet_train_step(pps_unet* u, int nx, int ny, int nz, const float* in_dev, const float* target_dev,
                               float lr, double* loss)
{
    if (!u || !in_dev || !target_dev || !loss || !(lr > 0.0f)) return PPS_ERR_INVALID_ARG;
    if (check_dims(nx, ny, nz) != PPS_OK) return PPS_ERR_INVALID_ARG;
    return uguard([&]() -> pps_status {
        UK(cudaSetDevice(u->device));
        loss_and_grads(u, nx, ny, nz, in_dev, target_dev);
        u->step += 1;
        rms((long long)u->npad, u->G, u->dtmp + 1, u->drms, u->stream);   // global-norm clipping at 1
        adam(u->pt, (int)u->npad, u->P, u->G, u->M, u->V, u->WP, u->WB, lr, 0.9f, 0.999f, 1e-8f, u->step, u->dtmp + 1,
             1.0f, u->stream);
        UK(cudaMemcpyAsync(loss, u->dloss, sizeof(double), cudaMemcpyDeviceToHost, u->stream));
        UK(cudaStreamSynchronize(u->stream));
        return PPS_OK;
    });
}

pps_status pps_restrict2(int nx, int ny, int nz, const float* fine_dev, float* coarse_dev)
{
    if (nx < 1 || ny < 1 || nz < 1 || ny > 32767 || nz > 32767 || !fine_dev || !coarse_dev) return PPS_ERR_INVALID_ARG;
    restrict2(Dims{nz, ny, nx}, fine_dev, coarse_dev, 0);
    return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? PPS_OK : PPS_ERR_CUDA;
}

pps_status pps_prolong2(int nx, int ny, int nz, const float* coarse_dev, float* fine_dev)
{
    if (nx < 1 || ny < 1 || nz < 1 || ny > 32767 || nz > 32767 || !fine_dev || !coarse_dev) return PPS_ERR_INVALID_ARG;
    prolong2(Dims{nz, ny, nx}, coarse_dev, fine_dev, 0);
    return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? PPS_OK : PPS_ERR_CUDA;
}

}  // extern "C"
