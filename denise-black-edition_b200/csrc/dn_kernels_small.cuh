// Velocity and elastic stress updates of the smallest batches (one-row tiles, up to about two
// tiles per resident block on the chip).
//
// The step of such a batch is bound by the chain of dependent memory round trips of one thread,
// each to L2 and back, not by bytes or instructions.  So every block copies its instance
// descriptor to shared memory in one round trip (the fields would otherwise be fetched line by
// line between the branches that need them); every operand of a row - the stencils, the row's own
// values, the CPML memory and its coefficients - is requested before any is used, with the
// registers that takes; and the launches overlap: a kernel starts while its predecessor drains
// (programmatic dependent launch), reads what no kernel writes (the descriptor, materials, CPML
// profiles) and waits for the predecessor before the first field.  Arithmetic and its order are
// those of the paired kernels, so results are the same bits.
//
// Measured against the folded paired kernels (2000 steps): 300 x 150, FDORDER 4: 27.3 -> 13.1 ms;
// 600 x 300, FDORDER 8: 30.1 -> 22.2 ms (its 1500 blocks are a quarter more than the 8 resident
// on each SM).  At 600 x 300 an SM issues in 28 % of its cycles and a warp waits 4.6 (velocity) and
// 5.7 (stress) issue slots for loads per instruction, DRAM and L2 far from their rates.  128 registers
// (8 blocks of 64 threads per SM) because with 80 or 64 the operands spill (300 x 150: 17.3 and
// 16.9 ms); requesting the lines into L1 first and loading late was slower still (27.6 ms).
#pragma once

#include "dn_kernels.cuh"

namespace dn {

// the predecessor's stores are visible after this; every block of a kernel launched with the
// programmatic attribute calls it, also a block without work (its end must not overtake them)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// the block's copy of its descriptor
__device__ __forceinline__ const Inst &stage_inst(const Inst *__restrict__ g, void *s)
{
    static_assert(sizeof(Inst) % 8 == 0, "descriptor copied in 8-byte words");
    const uint2 *src = reinterpret_cast<const uint2 *>(g);
    uint2 *dst = reinterpret_cast<uint2 *>(s);
    for (int k = threadIdx.x; k < (int)(sizeof(Inst) / 8); k += blockDim.x) dst[k] = __ldg(src + k);
    __syncthreads();
    return *reinterpret_cast<const Inst *>(s);
}

// CPML of a row's x frame for the two lanes of a pair (a frame narrower than half the grid, so
// that a column lies in one side at most): first the coefficients, then the memory, then the use.
struct XFrame2 {
    bool in[2];
    int h[2];
    float Ka[2], aa[2], ba[2], Kb[2], ab[2], bb[2], pa[2], pb[2];
    __device__ __forceinline__ void coefs(const Inst &I, int i0, const float *K1, const float *a1, const float *b1,
                                          const float *K2, const float *a2, const float *b2)
    {
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const int i = i0 + l;
            const bool left = i <= I.fw;
            in[l] = i <= I.nx && I.fw > 0 && (left || i >= I.nx - I.fw + 1);
            h[l] = left ? i - 1 : i - I.nx + 2 * I.fw - 1;
            if (in[l]) {
                Ka[l] = __ldg(K1 + h[l]), aa[l] = __ldg(a1 + h[l]), ba[l] = __ldg(b1 + h[l]);
                Kb[l] = __ldg(K2 + h[l]), ab[l] = __ldg(a2 + h[l]), bb[l] = __ldg(b2 + h[l]);
            }
        }
    }
    __device__ __forceinline__ void load(const Inst &I, int j, const float *psa, const float *psb)
    {
        const long long r = (long long)(j - 1) * 2 * I.fw;
#pragma unroll
        for (int l = 0; l < 2; l++)
            if (in[l]) pa[l] = psa[r + h[l]], pb[l] = psb[r + h[l]];
    }
    template <bool X>
    __device__ __forceinline__ void apply(const Inst &I, int j, float *psa, float *psb, float2 &da, float2 &db) const
    {
        const long long r = (long long)(j - 1) * 2 * I.fw;
        float *xa = &da.x, *xb = &db.x;
#pragma unroll
        for (int l = 0; l < 2; l++)
            if (in[l]) {
                const float v = ADD<X>(MUL<X>(ba[l], pa[l]), MUL<X>(aa[l], xa[l]));
                const float w = ADD<X>(MUL<X>(bb[l], pb[l]), MUL<X>(ab[l], xb[l]));
                psa[r + h[l]] = v;
                psb[r + h[l]] = w;
                xa[l] = ADD<X>(DIVK<X>(xa[l], Ka[l]), v);
                xb[l] = ADD<X>(DIVK<X>(xb[l], Kb[l]), w);
            }
    }
};
// the same for a row of the z frames
struct ZFrame2 {
    bool in;
    float Ka, aa, ba, Kb, ab, bb;
    float2 pa, pb;
    long long o;
    __device__ __forceinline__ void coefs(const Inst &I, int i0, int j, const float *K1, const float *a1, const float *b1,
                                          const float *K2, const float *a2, const float *b2)
    {
        const bool bottom = j >= I.ny - I.fw + 1;
        in = I.fw > 0 && ((!I.free_surf && j <= I.fw) || bottom);
        const int h = bottom ? j - I.ny + 2 * I.fw - 1 : j - 1;
        o = (long long)h * I.nx + (i0 - 1);
        if (in) {
            Ka = __ldg(K1 + h), aa = __ldg(a1 + h), ba = __ldg(b1 + h);
            Kb = __ldg(K2 + h), ab = __ldg(a2 + h), bb = __ldg(b2 + h);
        }
    }
    __device__ __forceinline__ void load(const float *psa, const float *psb, bool two)
    {
        if (!in) return;
        pa.x = psa[o], pb.x = psb[o];
        pa.y = two ? psa[o + 1] : 0.0f, pb.y = two ? psb[o + 1] : 0.0f;
    }
    template <bool X>
    __device__ __forceinline__ void apply(float *psa, float *psb, float2 &da, float2 &db, bool two) const
    {
        if (!in) return;
        const float *qa = &pa.x, *qb = &pb.x;
        float *xa = &da.x, *xb = &db.x;
#pragma unroll
        for (int l = 0; l < 2; l++) {
            if (l == 1 && !two) break;
            const float v = ADD<X>(MUL<X>(ba, qa[l]), MUL<X>(aa, xa[l]));
            const float w = ADD<X>(MUL<X>(bb, qb[l]), MUL<X>(ab, xb[l]));
            psa[o + l] = v;
            psb[o + l] = w;
            xa[l] = ADD<X>(DIVK<X>(xa[l], Ka), v);
            xb[l] = ADD<X>(DIVK<X>(xb[l], Kb), w);
        }
    }
};

// The pairs (k, k + 1), k = 0 .. 2R - 1, of an x stencil: KB the first aligned pair's index
template <int R, int KB>
__device__ __forceinline__ void pairs_load(const float *first, float2 *L)
{
#pragma unroll
    for (int q = 0; q <= R; q++) L[q] = ldw2(first + KB + 2 * q);
}
template <int R, int KB>
__device__ __forceinline__ float2 pair_at(const float2 *L, int k)
{
    if (((k - KB) & 1) == 0) return L[(k - KB) / 2];
    return make_float2(L[(k - 1 - KB) / 2].y, L[(k + 1 - KB) / 2].x);
}

// the source cell of a thread's pair, if any: its signal is requested with the row's operands
__device__ __forceinline__ bool small_source(const Inst &I, int i0, bool two, int j0, int j1, int nt)
{
    for (int c = 0; c < I.nsrc_cells; c++) {
        const int ci = I.sc_i[c], cj = I.sc_j[c];
        if (cj >= j0 && cj <= j1 && (ci == i0 || (two && ci == i0 + 1))) {
            const float *sg = I.signals + (long long)I.sc_l[c] * I.nt;
            pf_l1(sg + nt - 1);
            pf_l1(sg + max(nt - 2, 0));
            pf_l1(sg + min(nt, I.nt - 1));
            return true;
        }
    }
    return false;
}

template <int R, bool X>
__global__ void __launch_bounds__(64, 8) k_update_v2_small(const Inst *__restrict__ insts, const int *__restrict__ ntb, int off)
{
    __shared__ __align__(16) unsigned char s_inst[sizeof(Inst)];
    const int ntv = *ntb + off;   // written between graph launches only
    const Inst &I = stage_inst(insts + blockIdx.y, s_inst);
    pdl_launch();
    const int nt = ntv - I.t0;   // the instance's own time step
    const int b = blockIdx.x;
    const int tx = b % I.tiles_x, tz = b / I.tiles_x;
    const int i0 = tx * 2 * blockDim.x + 2 * threadIdx.x + 1;
    if (nt < 1 || nt > I.nt || b >= I.tiles || i0 > I.nx) {
        pdl_wait();
        return;
    }
    const int j0 = tz * I.zch + 1, j1 = min(j0 + I.zch - 1, I.ny);
    const bool two = i0 + 1 <= I.nx;
    const long long P = I.pitch;
    XFrame2 xf;
    xf.coefs(I, i0, I.K_xh, I.a_xh, I.b_xh, I.K_x, I.a_x, I.b_x);
    const bool snapstep = I.mode == 0 && I.store && ((nt - 1) % I.dtinv == 0);
    const bool fd = I.fastdiv;
    const float DT = I.DT, DH = I.DH, rdh = I.rdh;
    const bool srcs = I.fsrc_v && small_source(I, i0, two, j0, j1, nt);
    for (int j = j0; j <= j1; j++) {
        const long long o = (long long)j * P + i0;
        ZFrame2 zf;
        zf.coefs(I, i0, j, I.K_yh, I.a_yh, I.b_yh, I.K_y, I.a_y, I.b_y);
        const float2 ripv = ld2(I.rip + o), rjpv = ld2(I.rjp + o);
        if (j == j0) pdl_wait();
        constexpr int KA = (R % 2 == 0) ? -1 : 0, KX = (R % 2 == 0) ? 0 : -1;
        float2 la[R + 1], lx[R + 1], zy[2 * R], zx[2 * R];
        pairs_load<R, KA>(I.sxx + o - R + 1, la);
        pairs_load<R, KX>(I.sxy + o - R, lx);
#pragma unroll
        for (int k = 0; k < 2 * R; k++) {
            zy[k] = ldw2(I.syy + o + (k - R + 1) * P);   // rows j - R + 1 .. j + R
            zx[k] = ldw2(I.sxy + o + (k - R) * P);       // rows j - R .. j + R - 1
        }
        const float2 vxo = ldw2(I.vx + o), vyo = ldw2(I.vy + o);
        float2 p1x = make_float2(0.0f, 0.0f), p1y = p1x;
        if (I.mode == 1) p1x = ldw2(I.vxp1 + o), p1y = ldw2(I.vyp1 + o);
        xf.load(I, j, I.psi_sxx_x, I.psi_sxy_x);
        zf.load(I.psi_syy_y, I.psi_sxy_y, two);
        // derivatives, in the reference's term order (update_v_PML_PSV.c case 8 :366-480)
        float2 sxx_x = MUL2<X>(bc2(I.hc[1]), SUB2<X>(pair_at<R, KA>(la, R), pair_at<R, KA>(la, R - 1)));
        float2 sxy_x = MUL2<X>(bc2(I.hc[1]), SUB2<X>(pair_at<R, KX>(lx, R), pair_at<R, KX>(lx, R - 1)));
        float2 sxy_y = MUL2<X>(bc2(I.hc[1]), SUB2<X>(zx[R], zx[R - 1]));
        float2 syy_y = MUL2<X>(bc2(I.hc[1]), SUB2<X>(zy[R], zy[R - 1]));
#pragma unroll
        for (int m = 2; m <= R; m++) {
            const float2 h = bc2(I.hc[m]);
            sxx_x = ADD2<X>(sxx_x, MUL2<X>(h, SUB2<X>(pair_at<R, KA>(la, R - 1 + m), pair_at<R, KA>(la, R - m))));
            sxy_x = ADD2<X>(sxy_x, MUL2<X>(h, SUB2<X>(pair_at<R, KX>(lx, R + m - 1), pair_at<R, KX>(lx, R - m))));
            sxy_y = ADD2<X>(sxy_y, MUL2<X>(h, SUB2<X>(zx[R + m - 1], zx[R - m])));
            syy_y = ADD2<X>(syy_y, MUL2<X>(h, SUB2<X>(zy[R - 1 + m], zy[R - m])));
        }
        xf.apply<X>(I, j, I.psi_sxx_x, I.psi_sxy_x, sxx_x, sxy_x);
        zf.apply<X>(I.psi_syy_y, I.psi_sxy_y, syy_y, sxy_y, two);
        const float2 s1 = ADD2<X>(sxx_x, sxy_y);
        const float2 s2 = ADD2<X>(sxy_x, syy_y);
        float2 nvx = ADD2<X>(vxo, DIVH2<X>(MUL2<X>(MUL2<X>(bc2(DT), ripv), s1), fd, DH, rdh));
        float2 nvy = ADD2<X>(vyo, DIVH2<X>(MUL2<X>(MUL2<X>(bc2(DT), rjpv), s2), fd, DH, rdh));
        if (srcs) src_force_pair(I, i0, two, j, nt, nvx, nvy);
        if (snapstep) {
            p1x = DIVH2<X>(MUL2<X>(ripv, s1), fd, DH, rdh);
            p1y = DIVH2<X>(MUL2<X>(rjpv, s2), fd, DH, rdh);
        } else if (I.mode == 1) {
            p1x = ADD2<X>(p1x, MUL2<X>(bc2(DT), vxo));
            p1y = ADD2<X>(p1y, MUL2<X>(bc2(DT), vyo));
        }
        st2(I.vx + o, nvx, two);
        st2(I.vy + o, nvy, two);
        if (snapstep || I.mode == 1) {
            st2(I.vxp1 + o, p1x, two);
            st2(I.vyp1 + o, p1y, two);
        }
    }
}

template <int R, bool X>
__global__ void __launch_bounds__(64, 8) k_update_s_el2_small(const Inst *__restrict__ insts, const int *__restrict__ ntb, int off)
{
    __shared__ __align__(16) unsigned char s_inst[sizeof(Inst)];
    const int ntv = *ntb + off;   // written between graph launches only
    const Inst &I = stage_inst(insts + blockIdx.y, s_inst);
    pdl_launch();
    const int nt = ntv - I.t0;   // the instance's own time step
    const int b = (int)blockIdx.x - I.rec_blocks;
    const int tx = b % I.tiles_x, tz = b / I.tiles_x;
    const int i0 = tx * 2 * blockDim.x + 2 * threadIdx.x + 1;
    if (nt < 1 || nt > I.nt || b < 0 || b >= I.tiles || i0 > I.nx) {
        pdl_wait();
        if (nt >= 1 && nt <= I.nt && b < 0) record_velocities(I, nt, blockIdx.x, I.rec_blocks);
        return;
    }
    const int j0 = tz * I.zch + 1, j1 = min(j0 + I.zch - 1, I.ny);
    const bool two = i0 + 1 <= I.nx;
    const long long P = I.pitch;
    XFrame2 xf;
    xf.coefs(I, i0, I.K_x, I.a_x, I.b_x, I.K_xh, I.a_xh, I.b_xh);
    const bool srcs = I.fsrc_s && small_source(I, i0, two, j0, j1, nt);
    const int jsurf = I.surf_s ? R + 1 : 0;   // the last row with an image above the surface
    const float dhi = I.dhi_el;
    for (int j = j0; j <= j1; j++) {
        const long long o = (long long)j * P + i0;
        ZFrame2 zf;
        zf.coefs(I, i0, j, I.K_y, I.a_y, I.b_y, I.K_yh, I.a_yh, I.b_yh);
        const float2 fipjp = ld2(I.uipjp + o), f = ld2(I.mu + o), g = ld2(I.lam + o);
        if (j == j0) pdl_wait();
        constexpr int KC = (R % 2 == 0) ? 0 : -1, KD = (R % 2 == 0) ? -1 : 0;
        float2 lc[R + 1], ld[R + 1], zx[2 * R], zy[2 * R];
        pairs_load<R, KC>(I.vx + o - R, lc);
        pairs_load<R, KD>(I.vy + o - R + 1, ld);
#pragma unroll
        for (int k = 0; k < 2 * R; k++) {
            zx[k] = ldw2(I.vx + o + (k - R + 1) * P);   // rows j - R + 1 .. j + R
            zy[k] = ldw2(I.vy + o + (k - R) * P);       // rows j - R .. j + R - 1
        }
        const float2 s_xx = ldw2(I.sxx + o), s_yy = ldw2(I.syy + o), s_xy = ldw2(I.sxy + o);
        xf.load(I, j, I.psi_vxx, I.psi_vyx);
        if (jsurf && j == 1 && xf.in[0]) pf_l1(I.psi_vxxs + xf.h[0]);   // for the surface condition below
        zf.load(I.psi_vyy, I.psi_vxy, two);
        float2 vxx = MUL2<X>(bc2(I.hc[1]), SUB2<X>(pair_at<R, KC>(lc, R), pair_at<R, KC>(lc, R - 1)));
        float2 vyx = MUL2<X>(bc2(I.hc[1]), SUB2<X>(pair_at<R, KD>(ld, R), pair_at<R, KD>(ld, R - 1)));
        float2 vxy = MUL2<X>(bc2(I.hc[1]), SUB2<X>(zx[R], zx[R - 1]));
        float2 vyy = MUL2<X>(bc2(I.hc[1]), SUB2<X>(zy[R], zy[R - 1]));
#pragma unroll
        for (int m = 2; m <= R; m++) {
            const float2 h = bc2(I.hc[m]);
            vxx = ADD2<X>(vxx, MUL2<X>(h, SUB2<X>(pair_at<R, KC>(lc, R + m - 1), pair_at<R, KC>(lc, R - m))));
            vyx = ADD2<X>(vyx, MUL2<X>(h, SUB2<X>(pair_at<R, KD>(ld, R - 1 + m), pair_at<R, KD>(ld, R - m))));
            vxy = ADD2<X>(vxy, MUL2<X>(h, SUB2<X>(zx[R - 1 + m], zx[R - m])));
            vyy = ADD2<X>(vyy, MUL2<X>(h, SUB2<X>(zy[R + m - 1], zy[R - m])));
        }
        vxx = MUL2<X>(vxx, bc2(dhi));
        vyx = MUL2<X>(vyx, bc2(dhi));
        vxy = MUL2<X>(vxy, bc2(dhi));
        vyy = MUL2<X>(vyy, bc2(dhi));
        xf.apply<X>(I, j, I.psi_vxx, I.psi_vyx, vxx, vyx);
        zf.apply<X>(I.psi_vyy, I.psi_vxy, vyy, vxy, two);
        const float2 div = ADD2<X>(vxx, vyy);
        const float2 gdiv = MUL2<X>(g, div);
        const float2 nsxy = ADD2<X>(s_xy, MUL2<X>(fipjp, ADD2<X>(vyx, vxy)));
        float2 nsxx, nsyy;
        {
            const double f2x = 2.0 * (double)f.x, f2y = 2.0 * (double)f.y;
            nsxx.x = F(DADD((double)s_xx.x, DADD((double)gdiv.x, DMUL(f2x, (double)vxx.x))));
            nsxx.y = F(DADD((double)s_xx.y, DADD((double)gdiv.y, DMUL(f2y, (double)vxx.y))));
            nsyy.x = F(DADD((double)s_yy.x, DADD((double)gdiv.x, DMUL(f2x, (double)vyy.x))));
            nsyy.y = F(DADD((double)s_yy.y, DADD((double)gdiv.y, DMUL(f2y, (double)vyy.y))));
        }
        if (srcs) src_explosive_pair(I, i0, two, j, nt, nsxx, nsyy);
        if (j <= jsurf) {
            if (j == 1) {
                nsyy = make_float2(0.0f, 0.0f);
                nsxx.x = surface_sxx_el<R, X>(I, i0, o, nsxx.x);
                if (two) nsxx.y = surface_sxx_el<R, X>(I, i0 + 1, o + 1, nsxx.y);
            }
            surface_images<R>(I, j, o, nsyy.x, nsxy.x);
            if (two) surface_images<R>(I, j, o + 1, nsyy.y, nsxy.y);
        }
        st2(I.sxy + o, nsxy, two);
        st2(I.sxx + o, nsxx, two);
        st2(I.syy + o, nsyy, two);
    }
}

// launch with the programmatic attribute: the kernel may start while its predecessor drains
template <typename K>
static void launch_pdl(K kernel, dim3 grid, int block, cudaStream_t st, const Inst *d, const int *ntb, int off)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, d, ntb, off);
}

}   // namespace dn
