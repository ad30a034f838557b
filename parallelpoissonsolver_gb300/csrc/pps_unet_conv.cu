// Convolutions of the learned preconditioner's U-Net: forward, data gradient and
// weight gradient, with the elementwise steps between them folded into their loads
// and stores.  No reference counterpart.
//
// Activations are channels-last: act[((z*H + y)*W + x)*ld + c0 + c], BF16, where a
// tensor may occupy a channel slot [c0, c0+C) of a wider buffer (the U-Net's skip
// concatenations).  Convolutions are 3x3x3, zero-padded, stride 1, as implicit GEMMs
// on the tensor cores: M = voxels, N = output channels, K = 27 taps x input channels,
// m16n8k16 BF16 products with FP32 accumulators.
//
// The order of the sums is part of the network's definition: a BF16 activation whose
// FP32 sum rounds the other way differs by 2^-8, and such flips travel through all
// layers that follow (about 1e-4 of the output).  The K = 27 * Cin/16 steps are dealt
// round-robin to 8 chains (16 from 64 steps up), each summed in step order by the
// tensor core, and the chains are added in order; both kernels below keep exactly
// that, so which of them runs cannot be told from the result.  (Both run the
// same mma.sync products.  tcgen05 would need an accumulator for every chain, and whether
// its products round as these has not been measured.)
//
// Weights come packed in fragment order (k_pack, k_adam): one uint4 per lane holds a
// 16 x 16 block of W, so a step's weights are one coalesced 512-byte load.
#include "pps_unet_internal.h"

#include <algorithm>
#include <initializer_list>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace pps {
namespace unet {

namespace {

__device__ __forceinline__ float lo_f(unsigned w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(unsigned w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ unsigned pack_bf(float a, float b)
{
    return (unsigned)__bfloat16_as_ushort(__float2bfloat16(a)) |
           ((unsigned)__bfloat16_as_ushort(__float2bfloat16(b)) << 16);
}
// keep a channel where the layer's output y was positive (ReLU backward)
__device__ __forceinline__ unsigned relu_mask(unsigned v, unsigned y)
{
    return (lo_f(y) > 0.0f ? v & 0xffffu : 0u) | (hi_f(y) > 0.0f ? v & 0xffff0000u : 0u);
}

template <int NWORD>
struct Words {
    unsigned w[NWORD];
};
template <int NWORD>
__device__ __forceinline__ Words<NWORD> ld_words(const bf16* p)
{
    Words<NWORD> r;
    if constexpr (NWORD == 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(p);
        r.w[0] = q.x;
        r.w[1] = q.y;
        r.w[2] = q.z;
        r.w[3] = q.w;
    } else {
        r.w[0] = *reinterpret_cast<const unsigned*>(p);
    }
    return r;
}

// Channels [c, c + 2 NWORD) of the operand at voxel (z, y, x), which lies in the grid.
// in_sc: the scale of a dense source.
template <int NWORD, int KIND = -1>
__device__ __forceinline__ Words<NWORD> load_src(const Src& s, const Dims& d, int z, int y, int x, int c, float in_sc)
{
    const long long vox = ((long long)z * d.H + y) * d.W + x;
    const int kind = KIND >= 0 ? KIND : s.kind;   // known when the kernel was compiled, or uniform
    switch (kind) {
    case SRC_DENSE: {
        Words<NWORD> r;
#pragma unroll
        for (int q = 0; q < NWORD; q++) r.w[q] = 0u;
        if (c == 0) r.w[0] = (unsigned)__bfloat16_as_ushort(__float2bfloat16(s.dense[vox] * in_sc));
        return r;
    }
    case SRC_UP:
        if (c < s.c_up) {
            const long long cv = ((long long)(z >> 1) * (d.H / 2) + (y >> 1)) * (d.W / 2) + (x >> 1);
            return ld_words<NWORD>(s.up + cv * s.ld_up + c);
        }
        break;
    case SRC_SKIP: {
        Words<NWORD> r = ld_words<NWORD>(s.X + vox * s.ld + s.c0 + c), m;
        const long long cv = ((long long)(z >> 1) * (d.H / 2) + (y >> 1)) * (d.W / 2) + (x >> 1);
        const Words<NWORD> p = ld_words<NWORD>(s.up + cv * s.ld_up + c);
        if (s.mask) m = ld_words<NWORD>(s.mask + vox * s.ldm + c);
#pragma unroll
        for (int q = 0; q < NWORD; q++) {
            r.w[q] = pack_bf(lo_f(r.w[q]) + 0.125f * lo_f(p.w[q]), hi_f(r.w[q]) + 0.125f * hi_f(p.w[q]));
            if (s.mask) r.w[q] = relu_mask(r.w[q], m.w[q]);
        }
        return r;
    }
    default:
        break;
    }
    return ld_words<NWORD>(s.X + vox * s.ld + s.c0 + c);
}

__device__ __forceinline__ float src_scale(const Src& s)
{
    return s.kind == SRC_DENSE && s.rms ? (*s.rms > 0.0f ? 1.0f / *s.rms : 0.0f) : 1.0f;
}

__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// the same, kept in its place among the warp's shared-memory stores
__device__ __forceinline__ void ldsm4_ordered(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ldsm4t(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Pieces of `chunk` 16-byte words of a source into shared memory (asynchronous copies
// where the source is stored as the convolution reads it).
__device__ __forceinline__ void src_to_smem(const Src& s, const Dims& d, int z, int y, int x, int c, float in_sc,
                                            unsigned dst, unsigned char* dst_p, bool in)
{
    const bool plain = s.kind == SRC_PLAIN || s.kind == SRC_UP;
    if (plain && in) {
        const bf16* p;
        if (s.kind == SRC_UP && c < s.c_up)
            p = s.up + (((long long)(z >> 1) * (d.H / 2) + (y >> 1)) * (d.W / 2) + (x >> 1)) * s.ld_up + c;
        else
            p = s.X + (((long long)z * d.H + y) * d.W + x) * s.ld + s.c0 + c;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
        return;
    }
    uint4 v = make_uint4(0, 0, 0, 0);
    if (in) {
        const Words<4> w = load_src<4>(s, d, z, y, x, c, in_sc);
        v = make_uint4(w.w[0], w.w[1], w.w[2], w.w[3]);
    }
    *reinterpret_cast<uint4*>(dst_p) = v;
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// value of the loss term at voxel v and its gradient (MSE on channel 0)
__device__ __forceinline__ double mse_term(const Epi& e, long long v, float val)
{
    const float er = val - e.target[v];
    e.dense_out[v] = 2.0f * er * e.inv_n;
    return (double)er * (double)er;
}

}  // namespace

// ---------------------------------------------------------------------------
// Small grids.  One block: 16 consecutive voxels x 16 output channels, the K steps
// dealt to NW warps, so a block's dependent chain is 1/NW of K (a 16^3 grid has 256
// such blocks; latency, not the tensor pipe, is the limit).  A lane loads 8 channels of a
// voxel, four steps' loads in flight at a time, and a matrix load hands them out: loaded
// straight into the fragments, two channels at a time, they were twice the cache-line
// lookups, and layers of 48 and more channels were bound by those (forward on 16^3,
// 80/16/16 channels: 258 -> 184 us, 48/48/48 180 -> 137, 16/32/64 94 -> 84).
// ---------------------------------------------------------------------------
template <int NW, int KIND>
__global__ void __launch_bounds__(32 * NW) k_conv_small(Dims d, Src in, const uint4* __restrict__ Wp, int Cin, int Cout,
                                                        Epi e, const int* __restrict__ stop)
{
    pdl_enter();
    if (stop && *(volatile const int*)stop) return;
    constexpr int U = 4;
    __shared__ __align__(16) unsigned char buf[NW * U * 512];   // a warp's A blocks of U steps, then its sums
    __shared__ double sl[16];
    float (*sC)[16 * 16] = reinterpret_cast<float (*)[16 * 16]>(buf);
    const long long nvox = (long long)d.D * d.H * d.W;
    const long long v0 = (long long)blockIdx.x * 16;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    // the voxel whose channels this lane loads, the 8 of 16 it loads, and where they go: rows
    // of 32 bytes whose halves trade places every four rows, so that the eight rows of a
    // matrix load lie in different banks
    const int row = lane >> 1, half = lane & 1;
    const long long vox = v0 + row;
    const bool vin = vox < nvox;
    const int x = (int)(vox % d.W), y = (int)((vox / d.W) % d.H), z = (int)(vox / ((long long)d.W * d.H));
    unsigned char* const slot = buf + warp * (U * 512);
    unsigned char* const st = slot + row * 32 + ((half ^ (row >> 2)) & 1) * 16;
    const unsigned ld = smem_u32(slot) + (lane & 15) * 32 + (((lane >> 4) ^ ((lane & 15) >> 2)) & 1) * 16;
    const int csteps = Cin / 16, ksteps = 27 * csteps, n16 = Cout / 16;
    const float in_sc = src_scale(in);
    float acc[2][4] = {};
    for (int t0 = warp; t0 < ksteps; t0 += NW * U) {
        Words<4> a[U];
        uint4 b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int t = t0 + NW * u;
            a[u] = Words<4>{};
            b[u] = make_uint4(0, 0, 0, 0);
            if (t < ksteps) {
                b[u] = Wp[((long long)t * n16 + blockIdx.y) * 32 + lane];
                const int tap = t / csteps, c0 = (t - tap * csteps) * 16;
                const int zz = z + tap / 9 - 1, yy = y + (tap / 3) % 3 - 1, xx = x + tap % 3 - 1;
                if (vin && zz >= 0 && zz < d.D && yy >= 0 && yy < d.H && xx >= 0 && xx < d.W)
                    a[u] = load_src<4, KIND>(in, d, zz, yy, xx, c0 + 8 * half, in_sc);
            }
        }
        __syncwarp();   // the last round's matrix loads are done
#pragma unroll
        for (int u = 0; u < U; u++)
            *reinterpret_cast<uint4*>(st + u * 512) = make_uint4(a[u].w[0], a[u].w[1], a[u].w[2], a[u].w[3]);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; u++)
            if (t0 + NW * u < ksteps) {
                unsigned m[4];
                ldsm4_ordered(m, ld + u * 512);
                mma16816(acc[0], m, b[u].x, b[u].y);
                mma16816(acc[1], m, b[u].z, b[u].w);
            }
    }
    __syncthreads();   // the sums take the A blocks' place
#pragma unroll
    for (int n = 0; n < 2; n++) {
        *reinterpret_cast<float2*>(&sC[warp][gid * 16 + n * 8 + 2 * tig]) = make_float2(acc[n][0], acc[n][1]);
        *reinterpret_cast<float2*>(&sC[warp][(gid + 8) * 16 + n * 8 + 2 * tig]) = make_float2(acc[n][2], acc[n][3]);
    }
    __syncthreads();
    const int q = threadIdx.x;
    if (q < 256) {
        const int v = q >> 4, co = blockIdx.y * 16 + (q & 15);
        float val = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) val += sC[w][q];
        val += e.bias ? e.bias[co] : 0.0f;
        if (e.relu) val = fmaxf(val, 0.0f);
        const bool on = v0 + v < nvox;
        if (e.target) {
            if (co == 0) sl[v] = on ? mse_term(e, v0 + v, val) : 0.0;
        } else if (e.dense_out) {
            if (co == 0 && on) e.dense_out[v0 + v] = val * ((e.rms ? *e.rms : 1.0f) * e.gain);
        } else if (on) {
            bf16 r = __float2bfloat16(val);
            if (e.mask && !(__bfloat162float(e.mask[(v0 + v) * e.ldm + co]) > 0.0f)) r = __float2bfloat16(0.0f);
            e.Y[(v0 + v) * e.ld + co] = r;
        }
    }
    if (e.target) {
        __syncthreads();
        if (threadIdx.x == 0 && blockIdx.y == 0) {
            double s = 0.0;
            for (int v = 0; v < 16; v++) s += sl[v];
            atomicAdd(e.loss, s / (double)nvox);
        }
    }
}

// ---------------------------------------------------------------------------
// Large grids.  One block: a tile of 16 NWARP MG voxels x NC output channels.  The tile's
// input with its one-voxel halo is staged in shared memory once for all 27 taps
// (rows padded by 16 bytes, so the 8 rows of a matrix load hit different banks); a
// warp owns MG groups of 16 voxels and runs every K step itself, chain after chain, so
// a chain's accumulator lives in registers and the chains are added there in order.
// CS = Cin/16 and N16 = Cout/16 where they are known when compiled: the K loop then
// unrolls to matrix loads at fixed offsets (a table of steps in shared memory cost
// 18 instructions per product).  CS = 0: any channel counts, by the table.
// ---------------------------------------------------------------------------
template <int LX, int LY, int NWARP, int MG, int NC, int CS, int N16>
__global__ void __launch_bounds__(32 * NWARP, NWARP > 8 || NC == 48 ? 1 : 2) k_conv_tile(Dims d, Src in, const uint4* __restrict__ Wp, int Cin_,
                                                                     int Cout, Epi e, int chains_, int ntx, int nty,
                                                                     const int* __restrict__ stop)
{
    pdl_enter();
    if (stop && *(volatile const int*)stop) return;
    constexpr int TX = 1 << LX, TY = 1 << LY, TZ = (16 * NWARP * MG) >> (LX + LY);
    constexpr int HX = TX + 2, HY = TY + 2, HZ = TZ + 2, NB = NC / 16;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double sl[NWARP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Cin = CS > 0 ? CS * 16 : Cin_;
    const int stride = Cin * 2 + 16, nch = Cin / 8;
    const int csteps = Cin / 16, ksteps = 27 * csteps, n16 = N16 > 0 ? N16 : Cout / 16;
    int2* tab = reinterpret_cast<int2*>(smem + HX * HY * HZ * stride);   // K steps in chain order (CS = 0)
    const int bx = blockIdx.x % ntx, by = (blockIdx.x / ntx) % nty, bz = blockIdx.x / (ntx * nty);
    const int x0 = bx * TX, y0 = by * TY, z0 = bz * TZ;
    const unsigned sbase = smem_u32(smem);
    const float in_sc = src_scale(in);
    for (int q = tid; q < HX * HY * HZ * nch; q += 32 * NWARP) {
        const int v = q / nch, c = (q - v * nch) * 8;
        const int x = x0 - 1 + v % HX, y = y0 - 1 + (v / HX) % HY, z = z0 - 1 + v / (HX * HY);
        const bool ok = x >= 0 && x < d.W && y >= 0 && y < d.H && z >= 0 && z < d.D;
        const int o = v * stride + c * 2;
        src_to_smem(in, d, z, y, x, c, in_sc, sbase + o, smem + o, ok);
    }
    if (CS == 0 && tid < chains_) {
        // chain w holds steps w, w + chains, ...; the chains before it hold w whole rounds
        // of them, plus one more each for the first ksteps % chains
        const int w = tid, full = ksteps / chains_, rem = ksteps - full * chains_;
        int s = w * full + min(w, rem);
        for (int t = w; t < ksteps; t += chains_, s++) {
            const int tap = t / csteps, c0 = (t - tap * csteps) * 16;
            const int a = ((tap / 9) * HY + (tap / 3) % 3) * HX + tap % 3;
            tab[s] = make_int2((a * stride + c0 * 2) | (t + chains_ >= ksteps ? 1 : 0), t * n16 * 32);
        }
    }
    cp_wait_all();
    __syncthreads();

    // this lane's row of the warp's 16-voxel groups
    unsigned abase[MG];
#pragma unroll
    for (int m = 0; m < MG; m++) {
        const int r = (warp * MG + m) * 16 + (lane & 15);
        const int rx = r & (TX - 1), ry = (r >> LX) & (TY - 1), rz = r >> (LX + LY);
        abase[m] = sbase + ((rz * HY + ry) * HX + rx) * stride + (lane >> 4) * 16;
    }
    const uint4* wl = Wp + (long long)blockIdx.y * NB * 32 + lane;
    float tot[MG][2 * NB][4] = {}, acc[MG][2 * NB][4] = {};
    auto step = [&](int aoff, int boff) {
        uint4 b[NB];
#pragma unroll
        for (int n = 0; n < NB; n++) b[n] = wl[boff + n * 32];
#pragma unroll
        for (int m = 0; m < MG; m++) {
            unsigned a[4];
            ldsm4(a, abase[m] + aoff);
#pragma unroll
            for (int n = 0; n < NB; n++) {
                mma16816(acc[m][2 * n], a, b[n].x, b[n].y);
                mma16816(acc[m][2 * n + 1], a, b[n].z, b[n].w);
            }
        }
    };
    auto end_chain = [&]() {
#pragma unroll
        for (int m = 0; m < MG; m++)
#pragma unroll
            for (int n = 0; n < 2 * NB; n++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    tot[m][n][q] += acc[m][n][q];
                    acc[m][n][q] = 0.0f;
                }
    };
    if constexpr (CS > 0) {
        constexpr int KS = 27 * CS, CH = KS >= 64 ? 16 : 8;
#pragma unroll
        for (int w = 0; w < CH; w++) {
            // always taken (chains_ = CH), but the compiler does not know it: chains in one
            // basic block are interleaved, whose accumulators would not fit the registers
            if (w >= chains_) break;
#pragma unroll
            for (int t = w; t < KS; t += CH) {
                const int tap = t / CS, c0 = (t % CS) * 16;
                step((((tap / 9) * HY + (tap / 3) % 3) * HX + tap % 3) * (CS * 32 + 16) + c0 * 2, t * N16 * 32);
            }
            end_chain();
        }
    } else {
        int2 en = tab[0];
        for (int s = 0; s < ksteps; s++) {
            const int2 cur = en;
            if (s + 1 < ksteps) en = tab[s + 1];
            step(cur.x & ~1, cur.y);
            if (cur.x & 1) end_chain();
        }
    }
    const int gid = lane >> 2, tig = lane & 3, co0 = blockIdx.y * NC;
    double loss = 0.0;
#pragma unroll
    for (int m = 0; m < MG; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = (warp * MG + m) * 16 + gid + 8 * h;
            const int x = x0 + (r & (TX - 1)), y = y0 + ((r >> LX) & (TY - 1)), z = z0 + (r >> (LX + LY));
            if (x >= d.W || y >= d.H || z >= d.D) continue;
            const long long vox = ((long long)z * d.H + y) * d.W + x;
#pragma unroll
            for (int n = 0; n < 2 * NB; n++) {
                const int co = co0 + n * 8 + 2 * tig;
                float v0 = tot[m][n][2 * h], v1 = tot[m][n][2 * h + 1];
                v0 += e.bias ? e.bias[co] : 0.0f;
                v1 += e.bias ? e.bias[co + 1] : 0.0f;
                if (e.relu) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                }
                if (e.target) {
                    if (co == 0) loss += mse_term(e, vox, v0);
                } else if (e.dense_out) {
                    if (co == 0) e.dense_out[vox] = v0 * ((e.rms ? *e.rms : 1.0f) * e.gain);
                } else {
                    unsigned w = pack_bf(v0, v1);
                    if (e.mask) w = relu_mask(w, *reinterpret_cast<const unsigned*>(e.mask + vox * e.ldm + co));
                    *reinterpret_cast<unsigned*>(e.Y + vox * e.ld + co) = w;
                }
            }
        }
    if (e.target && co0 == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
        if (lane == 0) sl[warp] = loss;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < NWARP; w++) s += sl[w];
            atomicAdd(e.loss, s / ((double)d.D * d.H * d.W));
        }
    }
}

namespace {

// Tile shape of a grid: 256 voxels, as wide along x as the grid fills.
struct TileShape {
    int lx, ly, lz;
};
TileShape tile_shape(const Dims& d)
{
    if (d.W > 8) return TileShape{4, 2, 2};
    if (d.W > 4) return TileShape{3, 3, 2};
    return TileShape{2, 3, 3};
}
int ceil_div(int a, int b) { return (a + b - 1) / b; }

template <int LX, int LY, int NWARP, int MG, int NC, int CS, int N16>
void tile_launch(const Dims& d, const Src& in, const uint4* Wp, int Cin, int Cout, const Epi& e, int chains, cudaStream_t s)
{
    constexpr int TX = 1 << LX, TY = 1 << LY, TZ = (16 * NWARP * MG) >> (LX + LY);
    const int ntx = ceil_div(d.W, TX), nty = ceil_div(d.H, TY), ntz = ceil_div(d.D, TZ);
    const size_t smem = (size_t)(TX + 2) * (TY + 2) * (TZ + 2) * (Cin * 2 + 16) + (CS ? 0 : sizeof(int2) * 27 * (Cin / 16));
    launch_pdl(k_conv_tile<LX, LY, NWARP, MG, NC, CS, N16>, dim3((unsigned)(ntx * nty * ntz), (unsigned)(Cout / NC)),
               32 * NWARP, smem, s, d, in, Wp, Cin, Cout, e, chains, ntx, nty, stop_flag());
}

template <int LX, int LY>
void tile_any(const Dims& d, const Src& in, const uint4* Wp, int Cin, int Cout, const Epi& e, int chains, cudaStream_t s)
{
    if (Cout % 48 == 0) tile_launch<LX, LY, 8, 2, 48, 0, 0>(d, in, Wp, Cin, Cout, e, chains, s);
    else if (Cout % 32 == 0) tile_launch<LX, LY, 8, 2, 32, 0, 0>(d, in, Wp, Cin, Cout, e, chains, s);
    else tile_launch<LX, LY, 8, 2, 16, 0, 0>(d, in, Wp, Cin, Cout, e, chains, s);
}

// The 16-wide tiles of the default network's layers (channels 16/32/64), else any.
void tile_wide(const Dims& d, const Src& in, const uint4* Wp, int Cin, int Cout, const Epi& e, int chains, cudaStream_t s)
{
    const bool fills = (long long)d.D * d.H * d.W >= 512LL * sm_count();   // 512-voxel tiles for every SM
    switch (Cin * 100 + Cout) {
    case 1616: tile_launch<4, 3, 8, 4, 16, 1, 1>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 1632: tile_launch<4, 2, 8, 2, 32, 1, 2>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 1648: tile_launch<4, 2, 8, 2, 48, 1, 3>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 3216: tile_launch<4, 2, 8, 2, 16, 2, 1>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 3232: tile_launch<4, 2, 8, 2, 32, 2, 2>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 3264: tile_launch<4, 2, 8, 2, 32, 2, 4>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 3296: tile_launch<4, 2, 8, 2, 48, 2, 6>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 4816: tile_launch<4, 2, 8, 2, 16, 3, 1>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 6432: tile_launch<4, 2, 8, 2, 32, 4, 2>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 6464: tile_launch<4, 2, 8, 2, 32, 4, 4>(d, in, Wp, Cin, Cout, e, chains, s); break;
    case 9632:   // 135 KB a tile leaves one block per SM: sixteen warps of it where the grid has the tiles
        if (fills) tile_launch<4, 3, 16, 2, 32, 6, 2>(d, in, Wp, Cin, Cout, e, chains, s);
        else tile_launch<4, 2, 8, 2, 32, 6, 2>(d, in, Wp, Cin, Cout, e, chains, s);
        break;
    default: tile_any<4, 2>(d, in, Wp, Cin, Cout, e, chains, s); break;
    }
}

template <int KIND>
void small_launch(const Dims& d, const Src& in, const uint4* Wp, int Cin, int Cout, const Epi& e, int chains, cudaStream_t s)
{
    const dim3 grid((unsigned)(((long long)d.D * d.H * d.W + 15) / 16), (unsigned)(Cout / 16));
    if (chains == 16) launch_pdl(k_conv_small<16, KIND>, grid, 512, 0, s, d, in, Wp, Cin, Cout, e, stop_flag());
    else launch_pdl(k_conv_small<8, KIND>, grid, 256, 0, s, d, in, Wp, Cin, Cout, e, stop_flag());
}

cudaError_t allow_smem(std::initializer_list<const void*> kernels)
{
    cudaError_t e = cudaSuccess;
    for (const void* k : kernels)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    return e;
}
template <int LX, int LY>
cudaError_t allow_smem_any()
{
    return allow_smem({(const void*)k_conv_tile<LX, LY, 8, 2, 16, 0, 0>, (const void*)k_conv_tile<LX, LY, 8, 2, 32, 0, 0>,
                       (const void*)k_conv_tile<LX, LY, 8, 2, 48, 0, 0>});
}
cudaError_t allow_smem_wide()
{
    return allow_smem(
        {(const void*)k_conv_tile<4, 3, 8, 4, 16, 1, 1>, (const void*)k_conv_tile<4, 2, 8, 2, 32, 1, 2>,
         (const void*)k_conv_tile<4, 2, 8, 2, 48, 1, 3>, (const void*)k_conv_tile<4, 2, 8, 2, 16, 2, 1>,
         (const void*)k_conv_tile<4, 2, 8, 2, 32, 2, 2>, (const void*)k_conv_tile<4, 2, 8, 2, 32, 2, 4>,
         (const void*)k_conv_tile<4, 2, 8, 2, 48, 2, 6>, (const void*)k_conv_tile<4, 2, 8, 2, 16, 3, 1>,
         (const void*)k_conv_tile<4, 2, 8, 2, 32, 4, 2>, (const void*)k_conv_tile<4, 2, 8, 2, 32, 4, 4>,
         (const void*)k_conv_tile<4, 2, 8, 2, 32, 6, 2>, (const void*)k_conv_tile<4, 3, 16, 2, 32, 6, 2>});
}

}  // namespace

// Tiles of 256 voxels from which the tile kernel is the faster one (blocks of it that
// a launch needs to beat 16 times as many small ones).
constexpr int CONV_TILES_MIN = 32;

void conv(const Dims& d, const Src& in, const bf16* Wpacked, int Cin, int Cout, const Epi& e, cudaStream_t s)
{
    const int chains = 27 * (Cin / 16) >= 64 ? 16 : 8;
    const uint4* Wp = reinterpret_cast<const uint4*>(Wpacked);
    const TileShape t = tile_shape(d);
    const long long tiles = (long long)ceil_div(d.W, 1 << t.lx) * ceil_div(d.H, 1 << t.ly) * ceil_div(d.D, 1 << t.lz);
    if (tiles >= CONV_TILES_MIN) {
        if (t.lx == 4) tile_wide(d, in, Wp, Cin, Cout, e, chains, s);
        else if (t.lx == 3) tile_any<3, 3>(d, in, Wp, Cin, Cout, e, chains, s);
        else tile_any<2, 3>(d, in, Wp, Cin, Cout, e, chains, s);
    } else {
        switch (in.kind) {
        case SRC_PLAIN: small_launch<SRC_PLAIN>(d, in, Wp, Cin, Cout, e, chains, s); break;
        case SRC_DENSE: small_launch<SRC_DENSE>(d, in, Wp, Cin, Cout, e, chains, s); break;
        case SRC_UP: small_launch<SRC_UP>(d, in, Wp, Cin, Cout, e, chains, s); break;
        default: small_launch<SRC_SKIP>(d, in, Wp, Cin, Cout, e, chains, s); break;
        }
    }
    launches_counter_add(1);
}

// ---------------------------------------------------------------------------
// Weight and bias gradients of all layers in one launch:
//   dW[tap][ci][co] += sum_v X[v + off(tap)][ci] G[v][co],  db[co] += sum_v G[v][co].
// They depend on nothing but stored activations and gradients, so the 11 layers'
// work is one grid (the deep layers alone would fill a few blocks each).  One block:
// 16 input x up to 32 output channels over some tiles of 256 voxels, all 27 taps: warp
// w of 9 holds the taps (w/3, w%3, .) with FP32 accumulators in registers across the
// tiles, so X (with its halo) and G are read once per tile for 27 products, and the
// block adds to dW once.
// ---------------------------------------------------------------------------
constexpr int WG_THREADS = 288;
constexpr int WG_XSTRIDE = 48, WG_GSTRIDE = 80;   // bytes per voxel: 16 and 32 channels, padded by 16 bytes
constexpr int WG_HALO = 648;                      // the largest halo: 18 x 6 x 6 (10 x 10 x 6: 600)
constexpr int WG_SMEM = WG_HALO * WG_XSTRIDE + 256 * WG_GSTRIDE;

__global__ void __launch_bounds__(WG_THREADS, 2) k_wgrad(const __grid_constant__ WgTable T)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem[];
    int li = 0;
    while (li + 1 < T.n && (int)blockIdx.x >= T.L[li + 1].first) li++;
    const WgLayer& L = T.L[li];
    const Dims d = L.d;
    const int rel = blockIdx.x - L.first;
    const int kb = rel % L.kblocks, ci = (rel / L.kblocks) % (L.Cin / 16), cc = rel / (L.kblocks * (L.Cin / 16));
    const int nt = min(4, L.Cout / 8 - cc * 4);   // 8-channel tiles of G in this block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lx = L.lx, ly = L.ly, TX = 1 << lx, TY = 1 << ly, TZ = 256 >> (lx + ly);
    const int HX = TX + 2, HY = TY + 2, nhalo = HX * HY * (TZ + 2);
    unsigned char* sx = smem;
    unsigned char* sg = smem + WG_HALO * WG_XSTRIDE;
    const unsigned ax = smem_u32(sx), ag = smem_u32(sg);
    const float xsc = src_scale(L.X), gsc = src_scale(L.G);
    float acc[3][4][4] = {};
    float bsum = 0.0f;
    const int t1 = min((kb + 1) * L.tiles_per_block, L.ntx * L.nty * L.ntz);
    for (int t = kb * L.tiles_per_block; t < t1; t++) {
        const int x0 = (t % L.ntx) * TX, y0 = ((t / L.ntx) % L.nty) * TY, z0 = (t / (L.ntx * L.nty)) * TZ;
        __syncthreads();
        for (int q = tid; q < nhalo * 2; q += WG_THREADS) {
            const int v = q >> 1, c = (q & 1) * 8;
            const int x = x0 - 1 + v % HX, y = y0 - 1 + (v / HX) % HY, z = z0 - 1 + v / (HX * HY);
            const bool ok = x >= 0 && x < d.W && y >= 0 && y < d.H && z >= 0 && z < d.D;
            const int o = v * WG_XSTRIDE + c * 2;
            src_to_smem(L.X, d, z, y, x, ci * 16 + c, xsc, ax + o, sx + o, ok);
        }
        for (int q = tid; q < 256 * 4; q += WG_THREADS) {
            const int v = q >> 2, c = (q & 3) * 8;
            if (c >= nt * 8) continue;
            const int x = x0 + (v & (TX - 1)), y = y0 + ((v >> lx) & (TY - 1)), z = z0 + (v >> (lx + ly));
            const bool ok = x < d.W && y < d.H && z < d.D;
            const int o = v * WG_GSTRIDE + c * 2;
            src_to_smem(L.G, d, z, y, x, cc * 32 + c, gsc, ag + o, sg + o, ok);
        }
        cp_wait_all();
        __syncthreads();
        // lane's voxel of a 16-voxel step: rows of the transposed matrix loads
        const int av = (lane & 7) + ((lane >> 4) & 1) * 8, ac = ((lane >> 3) & 1) * 16;
        const int bv = (lane & 7) + ((lane >> 3) & 1) * 8, bc = (lane >> 4) * 16;
#pragma unroll 2
        for (int ks = 0; ks < 16; ks++) {
            unsigned b[2][4];
            ldsm4t(b[0], ag + (ks * 16 + bv) * WG_GSTRIDE + bc);
            if (nt > 2) ldsm4t(b[1], ag + (ks * 16 + bv) * WG_GSTRIDE + 32 + bc);
            const int r = ks * 16 + av;
            const int rx = r & (TX - 1), ry = (r >> lx) & (TY - 1), rz = r >> (lx + ly);
            const unsigned ar = ax + (((rz + warp / 3) * HY + ry + warp % 3) * HX + rx) * WG_XSTRIDE + ac;
#pragma unroll
            for (int dx = 0; dx < 3; dx++) {
                unsigned a[4];
                ldsm4t(a, ar + dx * WG_XSTRIDE);
                mma16816(acc[dx][0], a, b[0][0], b[0][1]);
                mma16816(acc[dx][1], a, b[0][2], b[0][3]);
                if (nt > 2) {
                    mma16816(acc[dx][2], a, b[1][0], b[1][1]);
                    mma16816(acc[dx][3], a, b[1][2], b[1][3]);
                }
            }
        }
        if (ci == 0 && lane < nt * 8) {   // bias: warp w sums rows w, w + 9, ... of column `lane`
            float b = 0.0f;
            for (int v = warp; v < 256; v += 9)
                b += __bfloat162float(*reinterpret_cast<const bf16*>(sg + v * WG_GSTRIDE + lane * 2));
            bsum += b;
        }
    }
    const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int dx = 0; dx < 3; dx++) {
        const int tap = warp * 3 + dx;
#pragma unroll
        for (int n = 0; n < 4; n++) {
            if (n >= nt) continue;
            float* p = L.dW + ((long long)tap * L.Cin + ci * 16 + gid) * L.Cout + cc * 32 + n * 8 + 2 * tig;
            atomicAdd(reinterpret_cast<float2*>(p), make_float2(acc[dx][n][0], acc[dx][n][1]));
            atomicAdd(reinterpret_cast<float2*>(p + 8LL * L.Cout), make_float2(acc[dx][n][2], acc[dx][n][3]));
        }
    }
    if (ci == 0) {   // the warps' sums first: one addition to db a block and channel
        float* sb = reinterpret_cast<float*>(smem);
        __syncthreads();
        sb[tid] = bsum;
        __syncthreads();
        if (tid < nt * 8) {
            float b = 0.0f;
            for (int w = 0; w < WG_THREADS / 32; w++) b += sb[w * 32 + tid];
            atomicAdd(&L.db[cc * 32 + tid], b);
        }
    }
}

void wgrad(WgTable& T, cudaStream_t s)
{
    // about two blocks per SM's worth of resident ones in all; a block's accumulators
    // cost 55 KB of atomics at its end, so it runs several tiles on large grids
    long long items = 0;
    for (int i = 0; i < T.n; i++) {
        WgLayer& L = T.L[i];
        const TileShape t = tile_shape(L.d);
        L.lx = t.lx;
        L.ly = t.ly;
        L.ntx = ceil_div(L.d.W, 1 << t.lx);
        L.nty = ceil_div(L.d.H, 1 << t.ly);
        L.ntz = ceil_div(L.d.D, 1 << t.lz);
        items += (long long)L.ntx * L.nty * L.ntz * (L.Cin / 16) * ceil_div(L.Cout, 32);
    }
    const long long target = 4LL * sm_count();
    const int per = (int)std::max(1LL, (items + target - 1) / target);
    int first = 0;
    for (int i = 0; i < T.n; i++) {
        WgLayer& L = T.L[i];
        // A block sums its tiles in one chain of the tensor core's FP32 accumulator, which
        // truncates, so the chain is bounded by the layer: half of a z plane's 16-voxel
        // steps, or the whole plane's up to 4 tiles.  Same-signed sums at 128^3 are off by
        // 5e-6 of their terms on the finest level and 6e-8 on the deepest; with `per` tiles
        // whatever the layer it was 8e-5 on both, in the same time (96% to 102%).
        const int plane = std::max(1, L.d.H * ceil_div(L.d.W, 16) / 16);   // tiles of 256 voxels
        const int chain = std::max(std::min(4, plane), plane / 2);
        L.tiles_per_block = std::min(per, chain);
        L.kblocks = ceil_div(L.ntx * L.nty * L.ntz, L.tiles_per_block);
        L.first = first;
        first += L.kblocks * (L.Cin / 16) * ceil_div(L.Cout, 32);
    }
    launch_pdl(k_wgrad, (unsigned)first, WG_THREADS, WG_SMEM, s, T);
    launches_counter_add(1);
}

// ---------------------------------------------------------------------------
// Sums over the 8 fine voxels of a coarse one: out[v][c] = BF16(scale * sum), kept where
// mask > 0.  scale 1/8: average pooling; scale 1: the gradient of a nearest upsampling.
// One thread per 8 channels.  (Folded into the convolution's loads instead, every
// output voxel repeats the 8 loads for each tap: 17 us for a 4^3 level against 3.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_gather8(Dims d, const bf16* __restrict__ X, int ld, int C, float scale,
                                                 const bf16* __restrict__ mask, bf16* __restrict__ out,
                                                 const int* __restrict__ stop)
{
    pdl_enter();
    if (stop && *(volatile const int*)stop) return;
    const int nch = C / 8;
    const long long n = (long long)d.D * d.H * d.W * nch;
    const long long Hf = 2LL * d.H, Wf = 2LL * d.W;
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < n; q += gridDim.x * 256LL) {
        const long long v = q / nch;
        const int c = (int)(q - v * nch) * 8;
        const int x = (int)(v % d.W), y = (int)((v / d.W) % d.H), z = (int)(v / ((long long)d.W * d.H));
        Words<4> w[8], r, m;
#pragma unroll
        for (int o = 0; o < 8; o++)
            w[o] = ld_words<4>(X + (((2LL * z + (o >> 2)) * Hf + 2 * y + ((o >> 1) & 1)) * Wf + 2 * x + (o & 1)) * ld + c);
        if (mask) m = ld_words<4>(mask + q * 8);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float a = 0.0f, b = 0.0f;
#pragma unroll
            for (int o = 0; o < 8; o++) {
                a += lo_f(w[o].w[k]);
                b += hi_f(w[o].w[k]);
            }
            r.w[k] = pack_bf(scale * a, scale * b);
            if (mask) r.w[k] = relu_mask(r.w[k], m.w[k]);
        }
        *reinterpret_cast<uint4*>(out + q * 8) = make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]);
    }
}

void gather8(const Dims& d, const bf16* X, int ld, int C, float scale, const bf16* mask, bf16* out, cudaStream_t s)
{
    const long long n = (long long)d.D * d.H * d.W * (C / 8);
    launch_pdl(k_gather8, (unsigned)std::min<long long>((n + 255) / 256, 16LL * sm_count()), 256, 0, s, d, X, ld, C, scale,
               mask, out, stop_flag());
    launches_counter_add(1);
}

// ---------------------------------------------------------------------------
// Parameters
// ---------------------------------------------------------------------------

// The packed copies of parameter q (a flat index of the padded master array): forward
// fragments at `fwd`, those of the data gradient (taps mirrored, channels swapped) at
// `bwd`.  A block of 16 x 16 weights [k][n] is one uint4 per lane: lane 4 (n % 8) +
// (k % 8) / 2 holds, for n < 8 and n >= 8, the pairs (k, k+1) of the lower and upper
// half of k.
__device__ __forceinline__ long long packed_at(int step, int k, int nblocks, int n)
{
    const int lane = (n & 7) * 4 + ((k & 7) >> 1);
    const int word = ((n >> 3) & 1) * 2 + (k >> 3);
    return ((((long long)step * nblocks + (n >> 4)) * 32 + lane) * 4 + word) * 2 + (k & 1);
}

__device__ __forceinline__ void pack_param(const PackTable& T, int q, float v, bf16* __restrict__ fwd,
                                           bf16* __restrict__ bwd)
{
    int l = 0;
    while (l + 1 < T.n && q >= T.w[l + 1]) l++;
    const int o = q - T.w[l], ci_n = T.cin[l], co_n = T.cout[l];
    if (o >= 27 * ci_n * co_n) return;   // a bias
    const int co = o % co_n, ci = (o / co_n) % ci_n, tap = o / (co_n * ci_n);
    const bf16 r = __float2bfloat16(v);
    fwd[T.w[l] + packed_at(tap * (ci_n / 16) + ci / 16, ci & 15, co_n / 16, co)] = r;
    bwd[T.w[l] + packed_at((26 - tap) * (co_n / 16) + co / 16, co & 15, ci_n / 16, ci)] = r;
}

__global__ void k_pack(const __grid_constant__ PackTable T, int n, const float* __restrict__ p, bf16* __restrict__ fwd,
                       bf16* __restrict__ bwd)
{
    pdl_enter();
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
        pack_param(T, q, p[q], fwd, bwd);
}

void pack(const PackTable& T, int n, const float* p, bf16* fwd, bf16* bwd, cudaStream_t s)
{
    launch_pdl(k_pack, (unsigned)((n + 255) / 256), 256, 0, s, T, n, p, fwd, bwd);
    launches_counter_add(1);
}

// Adam on FP32 master parameters; refreshes the packed BF16 copies of the weights.  The
// gradient is first scaled by min(1, max_norm / ||g||) (global-norm clipping), with
// ||g|| = (*g_rms) * sqrt(n) from k_rms.
__global__ void k_adam(const __grid_constant__ PackTable T, int n, float* __restrict__ p, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, bf16* __restrict__ fwd, bf16* __restrict__ bwd,
                       float lr, float b1, float b2, float eps, float c1, float c2, const float* g_rms, float max_norm)
{
    pdl_enter();
    float clip = 1.0f;
    const float norm = *g_rms * sqrtf((float)n);
    if (norm > max_norm && norm > 0.0f) clip = max_norm / norm;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const float gq = g[q] * clip;
        const float mq = b1 * m[q] + (1.0f - b1) * gq;
        const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        const float upd = lr * (mq / c1) / (sqrtf(vq / c2) + eps);
        const float pn = p[q] - upd;
        p[q] = pn;
        pack_param(T, q, pn, fwd, bwd);
    }
}

void adam(const PackTable& T, int n, float* p, const float* g, float* m, float* v, bf16* fwd, bf16* bwd, float lr,
          float b1, float b2, float eps, int step, const float* g_rms, float max_norm, cudaStream_t s)
{
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    launch_pdl(k_adam, (unsigned)((n + 255) / 256), 256, 0, s, T, n, p, g, m, v, fwd, bwd, lr, b1, b2, eps, c1, c2, g_rms,
               max_norm);
    launches_counter_add(1);
}

// rms of a dense FP32 array into *out: blocks of 1024 values a round, their FP64 sums
// in a fixed order, the last block to finish adds the blocks' (one block alone spent
// 206 us on the 367,216 gradients of a training step).
constexpr int RMS_BLOCKS = 256;
__global__ void __launch_bounds__(256) k_rms(long long n, const float* __restrict__ a, float* out, RmsScratch* sc,
                                             const int* __restrict__ stop)
{
    pdl_enter();
    if (stop && *(volatile const int*)stop) return;
    __shared__ double sm[8];
    __shared__ int is_last;
    const int tid = threadIdx.x;
    auto block_sum = [&](double s) -> double {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        __syncthreads();
        if ((tid & 31) == 0) sm[tid >> 5] = s;
        __syncthreads();
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += sm[w];
        return t;
    };
    double s = 0.0;
    for (long long q0 = (long long)blockIdx.x * 1024; q0 < n; q0 += (long long)gridDim.x * 1024) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = q0 + u * 256 + tid < n ? a[q0 + u * 256 + tid] : 0.0f;
#pragma unroll
        for (int u = 0; u < 4; u++) s += (double)v[u] * (double)v[u];
    }
    s = block_sum(s);
    if (tid == 0) {
        sc->part[blockIdx.x] = s;
        __threadfence();
        is_last = count_block(&sc->count, blockIdx.x, gridDim.x);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    s = block_sum(tid < (int)gridDim.x ? __ldcg(&sc->part[tid]) : 0.0);
    if (tid == 0) *out = (float)sqrt(s / (double)(n > 0 ? n : 1));
}

void rms(long long n, const float* a, float* out, RmsScratch* scratch, cudaStream_t s)
{
    const long long blocks = std::min<long long>(RMS_BLOCKS, std::max<long long>(1, (n + 1023) / 1024));
    launch_pdl(k_rms, (unsigned)blocks, 256, 0, s, n, a, out, scratch, stop_flag());
    launches_counter_add(1);
}

cudaError_t conv_prepare()
{
    cudaError_t e = allow_smem_any<4, 2>();
    if (e == cudaSuccess) e = allow_smem_any<3, 3>();
    if (e == cudaSuccess) e = allow_smem_any<2, 3>();
    if (e == cudaSuccess) e = allow_smem_wide();
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, WG_SMEM);
    return e;
}

}  // namespace unet
}  // namespace pps
