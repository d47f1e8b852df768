// potential.cu -- N^2 potential behind the reference's gpupot_ C ABI
// (gpupot.gpu.cu:116-127): pot[k] = sum_{j: r2 > 0} m_j / r_ij for
// i = istart-1+k, k in [0, ni).
//
// The j set (m, x) is copied once per call into device buffers that persist
// across calls (the reference allocates and frees per call,
// gpupot.gpu.cu:72-79,107-108), split into hi/lo FP32 rows laid out tile by
// tile, and streamed through a 4-stage ring of bulk copies, one per 128-j
// tile.  Each thread holds NI i-particles; pair math is packed FP32 (two j per
// f32x2 instruction) on hi/lo differences with rsqrt + one Newton step, FP32
// partial sums fold into double-single accumulators per tile, slices are
// summed in FP64 in a fixed order.  Large calls order the bodies in space
// first, so that most tiles are far from a whole warp's i-particles and take
// a shorter loop (pot_kernel).
#include "nb6_common.cuh"
#include "spatial.cuh"

#include <algorithm>
#include <string.h>

namespace {

constexpr int JT = 128;
constexpr int NSTAGE = 4;
constexpr int NT = 128;
constexpr unsigned long long WAIT_NS = 2000000000ull;

// Rows of one 128-body tile, JT floats each: xh, yh, zh, m, xl, yl, zl and,
// for an ordered set, xr, yr, zr (positions relative to the tile's box
// centre).  A tile is one contiguous block, so one bulk copy brings it in.
constexpr int ROWS_HL = 7, ROWS_ORD = 10;

// The call whose pairs number at least POT_ORDER_PAIRS, against a set of at
// least POT_ORDER_MIN bodies, orders the set: the order costs about 80 us at
// 131,071 bodies, and a far pair takes half the time of a near one.  (32,767 of
// 131,071 bodies, 4.3e9 pairs: 3,017 us as a scalar loop over the unordered
// set, 1,480 us ordered and packed, the order included.)  A far pair has one
// FP32 difference and no Newton step, yet the sums are no further off than the
// scalar loop's over hi/lo differences, which folded 128 terms at a time: on
// ranges of 1/8 to 1/2 of 45,000 to 239,999 bodies 0.8-1.3e-8 of the potential
// (2-norm) against 1.5-1.8e-8, on sets with heavy bodies, two clumps, a distant
// origin or one shell 0.8-12e-8 against 1.5-33e-8.
constexpr int POT_ORDER_MIN = 32768;
constexpr double POT_ORDER_PAIRS = 1.0e9;

struct PotArgs {
    const float *__restrict__ tiles;  // [ntile][rows][JT]
    const float4 *__restrict__ tbox;  // ordered: per tile (centre, 0), (half extents, 0)
    const double *__restrict__ x;     // FP64 positions [n][3], caller's order
    const int *__restrict__ idx;      // i-particle of slot k; null: body i0 + k
    int ntile, nslices;
    int i0, ni;                       // absolute first i (0-based), count
    float2 *__restrict__ part;        // [nslices][ni] (hi, lo) over slots
    int *status;
};

NB6_DEV float2 pair2(float v) { return make_float2(v, v); }
NB6_DEV float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
NB6_DEV float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }
NB6_DEV float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

NB6_DEV float2 rsqrt_approx2(float2 r2) {
    float2 y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(r2.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(r2.y));
    return y;
}

// sum -2 m / r over two j's into acc (lane = j parity), hi/lo differences
NB6_DEV void near_pair(float2 xh, float2 yh, float2 zh, float2 m, float2 xl, float2 yl, float2 zl, float2 nxh,
                       float2 nyh, float2 nzh, float2 nxl, float2 nyl, float2 nzl, float2 &acc) {
    const float2 dx = __fadd2_rn(__fadd2_rn(xh, nxh), __fadd2_rn(xl, nxl));
    const float2 dy = __fadd2_rn(__fadd2_rn(yh, nyh), __fadd2_rn(yl, nyl));
    const float2 dz = __fadd2_rn(__fadd2_rn(zh, nzh), __fadd2_rn(zl, nzl));
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    const float2 y0 = rsqrt_approx2(r2);
    const float2 nb = __ffma2_rn(__fmul2_rn(r2, y0), y0, pair2(-3.0f));  // -(3 - r2 y0^2)
    float2 ny = __fmul2_rn(y0, nb);                                      // -2/r
    ny.x = r2.x > 0.f ? ny.x : 0.f;  // gpupot.gpu.cu:52 skips r2 == 0
    ny.y = r2.y > 0.f ? ny.y : 0.f;
    acc = __ffma2_rn(m, ny, acc);
}

// sum m / r over two j's of a far tile: tile-relative differences, and 1/r
// straight from rsqrt.approx: every term of the sum is positive, so its
// relative error bound carries over to the sum unamplified (no Newton step
// needed, unlike the cancelling force sums).
NB6_DEV void far_pair(float2 xr, float2 yr, float2 zr, float2 m, float2 nxr, float2 nyr, float2 nzr, float2 &acc) {
    const float2 dx = __fadd2_rn(xr, nxr);
    const float2 dy = __fadd2_rn(yr, nyr);
    const float2 dz = __fadd2_rn(zr, nzr);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    acc = __ffma2_rn(m, rsqrt_approx2(r2), acc);
}

// One CTA: NT * NI i-particles against the tiles slice, slice + nslices, ...
// (the near tiles of a compact group of i are dealt out among the slices).
//
// ORD (bodies in Morton order with one bounding box per tile): a (warp, tile)
// whose box is at least one half extent away from every lane's i takes the
// far loop: differences from tile-relative coordinates fl32(x_j - c) (stored)
// and fl32(x_i - c) (formed in FP64 per tile), one FP32 add each instead of
// three, within 4 FP32 ulps of the FP64-formed difference (|x_j - c| <= h
// <= r).  Other tiles take the hi/lo loop.
//
// What bounds it: a far pair costs 7 FMA-pipe lane operations and one MUFU
// rsqrt, i.e. 1.75 and 2 cycles of an SM per warp and j, so the MUFU rate
// (16 lanes per cycle) is the floor.  One shared-memory load of 16 bytes per
// lane costs two cycles as well, and the loop needs one per j: with one i per
// thread the load path was 70% busy and the MUFU 64%.  Two i per thread
// (NI = 2, 96 registers, five CTAs per SM) share each load.  Warps release a
// stage on its own "empty" barrier, so they drift apart instead of meeting at
// a CTA barrier per tile.  249,036 bodies of a King cluster: 20.8 ms before
// (64% of the MUFU floor), 18.0 ms with one i per thread, 17.3 ms with two.
template <int NI, bool ORD>
__global__ void __launch_bounds__(NT, NI == 2 ? 5 : 8) pot_kernel(const PotArgs a) {
    constexpr int ROWS = ORD ? ROWS_ORD : ROWS_HL;
    constexpr uint32_t TILE_BYTES = ROWS * JT * sizeof(float);
    __shared__ __align__(128) float sj[NSTAGE][ROWS][JT];
    __shared__ __align__(8) uint64_t bar[NSTAGE], ebar[NSTAGE];
    const int tid = threadIdx.x, lane = tid & 31;
    const int slice = blockIdx.y;
    const int nt = slice < a.ntile ? (a.ntile - slice + a.nslices - 1) / a.nslices : 0;

    double xd[NI], yd[NI], zd[NI];
    float ph[NI], pl[NI];
    bool on[NI];
#pragma unroll
    for (int k = 0; k < NI; ++k) {
        const int s = blockIdx.x * (NT * NI) + k * NT + tid;
        on[k] = s < a.ni;
        xd[k] = yd[k] = zd[k] = 0.0;
        ph[k] = pl[k] = 0.f;
        if (on[k]) {
            const double *p = a.x + 3 * (size_t)(a.idx ? a.idx[s] : a.i0 + s);
            xd[k] = p[0];
            yd[k] = p[1];
            zd[k] = p[2];
        }
    }
    if (tid == 0) {
#pragma unroll
        for (int st = 0; st < NSTAGE; ++st) {
            mbar_init(&bar[st], 1);
            mbar_init(&ebar[st], NT / 32);
        }
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int t) {
        const int st = t % NSTAGE;
        mbar_arrive_expect_tx(&bar[st], TILE_BYTES);
        bulk_g2s(sj[st], a.tiles + (size_t)(slice + t * a.nslices) * (ROWS * JT), TILE_BYTES, &bar[st]);
    };
    int issued = 0;  // thread 0 only
    if (tid == 0)
        for (; issued < min(nt, NSTAGE); ++issued) issue(issued);

    for (int t = 0; t < nt; ++t) {
        const int st = t % NSTAGE;
        const uint32_t par = (uint32_t)((t / NSTAGE) & 1);
        if (!__all_sync(0xffffffffu, mbar_wait_timed(&bar[st], par, WAIT_NS))) {
            set_status(a.status, NB6_ERR_WAIT_TIMEOUT);
            if (tid == 0)  // drain copies still in flight before the CTA's smem goes away
                for (int u = t; u < issued; ++u)
                    mbar_wait_timed(&bar[u % NSTAGE], (uint32_t)((u / NSTAGE) & 1), WAIT_NS / 8);
            return;
        }
        const float(*S)[JT] = sj[st];
        bool far = false;
        float4 bc;
        if constexpr (ORD) {
            const int tile = slice + t * a.nslices;
            bc = __ldg(&a.tbox[2 * tile]);
            const float4 bh = __ldg(&a.tbox[2 * tile + 1]);
            // far: the box at least one half extent from this thread's i
            // (with a margin for the FP32 test); padding slots are far
            const float hm = fmaxf(fmaxf(bh.x, bh.y), bh.z);
            bool f = true;
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                const float ex = fmaxf(fabsf((float)xd[k] - bc.x) - bh.x, 0.f);
                const float ey = fmaxf(fabsf((float)yd[k] - bc.y) - bh.y, 0.f);
                const float ez = fmaxf(fabsf((float)zd[k] - bc.z) - bh.z, 0.f);
                f = f && (!on[k] || ex * ex + ey * ey + ez * ez > 1.01f * hm * hm);
            }
            far = __all_sync(0xffffffffu, f);
        }
        float2 acc[NI];
#pragma unroll
        for (int k = 0; k < NI; ++k) acc[k] = make_float2(0.f, 0.f);
        if (ORD && far) {
            float2 nx[NI], ny[NI], nz[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                nx[k] = pair2(-__double2float_rn(xd[k] - (double)bc.x));
                ny[k] = pair2(-__double2float_rn(yd[k] - (double)bc.y));
                nz[k] = pair2(-__double2float_rn(zd[k] - (double)bc.z));
            }
#pragma unroll 8
            for (int q = 0; q < JT; q += 4) {
                const float4 M = ld4(&S[3][q]), X = ld4(&S[ROWS - 3][q]), Y = ld4(&S[ROWS - 2][q]),
                             Z = ld4(&S[ROWS - 1][q]);
#pragma unroll
                for (int k = 0; k < NI; ++k) {
                    far_pair(lo2(X), lo2(Y), lo2(Z), lo2(M), nx[k], ny[k], nz[k], acc[k]);
                    far_pair(hi2(X), hi2(Y), hi2(Z), hi2(M), nx[k], ny[k], nz[k], acc[k]);
                }
            }
        } else {
            float2 nxh[NI], nyh[NI], nzh[NI], nxl[NI], nyl[NI], nzl[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                float h, l;
                split_hl(xd[k], h, l);
                nxh[k] = pair2(-h);
                nxl[k] = pair2(-l);
                split_hl(yd[k], h, l);
                nyh[k] = pair2(-h);
                nyl[k] = pair2(-l);
                split_hl(zd[k], h, l);
                nzh[k] = pair2(-h);
                nzl[k] = pair2(-l);
            }
#pragma unroll 4
            for (int q = 0; q < JT; q += 4) {
                const float4 XH = ld4(&S[0][q]), YH = ld4(&S[1][q]), ZH = ld4(&S[2][q]), M = ld4(&S[3][q]),
                             XL = ld4(&S[4][q]), YL = ld4(&S[5][q]), ZL = ld4(&S[6][q]);
#pragma unroll
                for (int k = 0; k < NI; ++k) {
                    near_pair(lo2(XH), lo2(YH), lo2(ZH), lo2(M), lo2(XL), lo2(YL), lo2(ZL), nxh[k], nyh[k], nzh[k],
                              nxl[k], nyl[k], nzl[k], acc[k]);
                    near_pair(hi2(XH), hi2(YH), hi2(ZH), hi2(M), hi2(XL), hi2(YL), hi2(ZL), nxh[k], nyh[k], nzh[k],
                              nxl[k], nyl[k], nzl[k], acc[k]);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ebar[st]);
        if (tid == 0 && issued < nt) {
            // once every warp has released tile t, refill its stage
            if (!mbar_wait_timed(&ebar[st], par, WAIT_NS)) {
                set_status(a.status, NB6_ERR_WAIT_TIMEOUT);
                for (int u = t + 1; u < issued; ++u)
                    mbar_wait_timed(&bar[u % NSTAGE], (uint32_t)((u / NSTAGE) & 1), WAIT_NS / 8);
                return;
            }
            issue(issued);
            ++issued;
        }
        const float f = far ? 1.0f : -0.5f;
#pragma unroll
        for (int k = 0; k < NI; ++k) ds_fold(ph[k], pl[k], f * (acc[k].x + acc[k].y));
    }
#pragma unroll
    for (int k = 0; k < NI; ++k) {
        const int s = blockIdx.x * (NT * NI) + k * NT + tid;
        if (on[k]) a.part[(size_t)slice * a.ni + s] = make_float2(ph[k], pl[k]);
    }
}

// Sum of the slices of slot k, in order, to out[idx[k] - i0] (the caller's
// index) or out[k].  hstatus: see nb6_status_post.
__global__ void pot_finalize(const float2 *__restrict__ part, int nslices, int i0, int ni,
                             const int *__restrict__ idx, double *__restrict__ out, const int *status,
                             int *hstatus, DevSpan *span) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (hstatus && k == 0) *hstatus = *status;
    if (k >= ni) return;
    double v = 0.0;
#pragma unroll 8
    for (int sl = 0; sl < nslices; ++sl) {
        const float2 p = __ldg(part + (size_t)sl * ni + k);
        v += (double)p.x + (double)p.y;
    }
    out[idx ? idx[k] - i0 : k] = v;
    if (span && threadIdx.x == 0) span_end(span);
}

// One CTA per tile: its rows of the tile layout, from the bodies in the
// caller's order (ROWS_HL) or, with perm, in Morton order, with the tile's
// box (of the hi positions of its real bodies: centre rounded to nearest,
// half extents rounded up) and the tile-relative rows.  Padding slots are
// massless and far away.  keep not null: m and x are in pinned host memory,
// and a copy of x is kept on the device.
template <bool ORD>
__global__ void __launch_bounds__(JT) pot_tiles(int n, const int *__restrict__ perm, const double *__restrict__ m,
                                                const double *__restrict__ x, double *__restrict__ keep,
                                                float *__restrict__ tiles, float4 *__restrict__ tbox, int *status,
                                                DevSpan *span) {
    constexpr int ROWS = ORD ? ROWS_ORD : ROWS_HL;
    const int t = threadIdx.x, s = blockIdx.x * JT + t;
    if (span && s == 0) span_begin(span);
    double c[3] = {1.0e15, 1.0e15, 1.0e15}, mj = 0.0;
    if (s < n) {
        const size_t j = ORD ? perm[s] : s;
#pragma unroll
        for (int k = 0; k < 3; ++k) c[k] = x[3 * j + k];
        mj = m[j];
        if (keep)
#pragma unroll
            for (int k = 0; k < 3; ++k) keep[3 * j + k] = c[k];
        if (c[0] != c[0] || c[1] != c[1] || c[2] != c[2] || mj != mj) set_status(status, NB6_ERR_NAN_INPUT);
    }
    float *o = tiles + (size_t)blockIdx.x * (ROWS * JT) + t;
    float h[3], l[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        split_hl(c[k], h[k], l[k]);
        o[k * JT] = h[k];
        o[(4 + k) * JT] = l[k];
    }
    o[3 * JT] = (float)mj;
    if constexpr (ORD) {
        __shared__ unsigned smn[JT / 32][3], smx[JT / 32][3];
        __shared__ float sc[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned u = f2ord(h[k]);
            const unsigned mn = __reduce_min_sync(0xffffffffu, s < n ? u : 0xffffffffu);
            const unsigned mx = __reduce_max_sync(0xffffffffu, s < n ? u : 0u);
            if ((t & 31) == 0) {
                smn[t >> 5][k] = mn;
                smx[t >> 5][k] = mx;
            }
        }
        __syncthreads();
        if (t < 3) {
            unsigned a = smn[0][t], b = smx[0][t];
            for (int w = 1; w < JT / 32; ++w) {
                a = min(a, smn[w][t]);
                b = max(b, smx[w][t]);
            }
            const double lo = ord2f(a), hi = ord2f(b);
            sc[t] = __double2float_rn(0.5 * (lo + hi));
            float *bx = reinterpret_cast<float *>(tbox + 2 * blockIdx.x);
            bx[t] = sc[t];
            bx[4 + t] = __double2float_ru(0.5 * (hi - lo));
            if (t == 0) bx[3] = bx[7] = 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; ++k) o[(7 + k) * JT] = __double2float_rn(c[k] - (double)sc[k]);
    }
}

// The bodies [i0, i0+ni) of an ordered set, in that order: idx[k] = the k-th
// slot's body, among the slots whose body is in the range.  Two launches:
// counts per CTA, then each CTA adds up the counts before its own and packs
// its slots.
constexpr int SEL_NT = 1024;
__global__ void __launch_bounds__(SEL_NT) pot_select_count(int n, const int *__restrict__ perm, int i0, int ni,
                                                           int *__restrict__ count) {
    const int s = blockIdx.x * SEL_NT + threadIdx.x;
    const int c = __syncthreads_count(s < n && (unsigned)(perm[s] - i0) < (unsigned)ni);
    if (threadIdx.x == 0) count[blockIdx.x] = c;
}

__global__ void __launch_bounds__(SEL_NT) pot_select(int n, const int *__restrict__ perm, int i0, int ni,
                                                     const int *__restrict__ count, int *__restrict__ idx) {
    __shared__ int wsum[SEL_NT / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int s = blockIdx.x * SEL_NT + t;
    const int body = s < n ? perm[s] : -1;
    const bool in = s < n && (unsigned)(body - i0) < (unsigned)ni;
    const unsigned b = __ballot_sync(0xffffffffu, in);
    int before = 0;
    for (int q = t; q < (int)blockIdx.x; q += SEL_NT) before += count[q];
    // this warp's share of the counts before the CTA, plus its own slots
    const int share = __reduce_add_sync(0xffffffffu, before);
    __shared__ int base[SEL_NT / 32];
    if (lane == 0) {
        base[warp] = share;
        wsum[warp] = __popc(b);
    }
    __syncthreads();
    int off = 0;
    for (int w = 0; w < SEL_NT / 32; ++w) off += base[w] + (w < warp ? wsum[w] : 0);
    if (in) idx[off + __popc(b & ((1u << lane) - 1u))] = body;
}

struct PotState {
    DevBuf<double> mx, out;                     // the bodies of a host call: m, x
    DevBuf<float> tiles;
    DevBuf<float4> tbox;
    DevBuf<float2> part;
    DevBuf<int> count, idx;
    HostBuf<double> hout;
    SpatialOrder order;
    int n = 0, ntile = 0;
    const double *dm = nullptr, *dx = nullptr;  // the m, x of the call, readable by kernels
    double *keep = nullptr;                     // where to keep x when dx is pinned host memory
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;   // an ordered call's time; an unordered one stamps its own
    DevBuf<DevSpan> span;
    bool stamped = false;
    float last_ms = 0.f;
};
PotState P;

// Whether a call orders its set (NB6_POT_ORDER=0: never).
bool pot_ordered(int ni) {
    static const int ordered = [] {
        const char *e = getenv("NB6_POT_ORDER");
        return (e && atoi(e) == 0) ? 0 : 1;
    }();
    return ordered && P.n >= POT_ORDER_MIN && (double)P.n * ni >= POT_ORDER_PAIRS;
}

template <int NI, bool ORD> int pot_occ() {
    static const int occ = [] {
        int o = 0;
        NB6_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, pot_kernel<NI, ORD>, NT, 0));
        return std::max(o, 1);
    }();
    return occ;
}

// Slices per i-tile.  A call that fills the GPU is cut into about six waves
// of CTAs, so that the last one leaves little idle, each of at least 16 tiles
// (its set-up costs about half a tile); a small one into one wave.
template <int NI, bool ORD> void pot_launch(PotArgs &a, cudaStream_t st) {
    const int nitile = (a.ni + NT * NI - 1) / (NT * NI);
    const int slots = nb6_num_sms() * pot_occ<NI, ORD>();
    const int one_wave = std::max(1, slots / nitile), six_waves = (6 * slots + nitile - 1) / nitile;
    a.nslices = std::min(std::max(one_wave, std::min(six_waves, a.ntile / 16)), a.ntile);
    P.part.reserve((size_t)a.nslices * a.ni);
    a.part = P.part.ptr;
    pot_kernel<NI, ORD><<<dim3(nitile, a.nslices), NT, 0, st>>>(a);
    NB6_CUDA_CHECK(cudaGetLastError());
}

// Potential of i in [i0, i0+ni) of the uploaded bodies (P.dm, P.dx, P.n).
// The result goes to hout (pinned, with the status word posted) when the
// call writes it in the caller's order, else to P.out; returns whether it
// went to hout.
bool pot_compute(int i0, int ni, double *hout, cudaStream_t st) {
    const int n = P.n;
    PotArgs a{};
    a.x = P.keep ? P.keep : P.dx;
    a.ntile = P.ntile;
    a.i0 = i0;
    a.ni = ni;
    a.status = nb6_dev_status();
    const bool ord = pot_ordered(ni);
    P.tiles.reserve((size_t)P.ntile * (ord ? ROWS_ORD : ROWS_HL) * JT);
    a.tiles = P.tiles.ptr;
    if (ord) {
        P.order.build(n, P.dx, st);
        P.tbox.reserve(2 * (size_t)P.ntile);
        pot_tiles<true><<<P.ntile, JT, 0, st>>>(n, P.order.perm.ptr, P.dm, P.dx, nullptr, P.tiles.ptr, P.tbox.ptr,
                                                a.status, nullptr);
        NB6_CUDA_CHECK(cudaGetLastError());
        a.tbox = P.tbox.ptr;
        a.idx = P.order.perm.ptr;
        if (ni < n) {
            const int sb = (n + SEL_NT - 1) / SEL_NT;
            P.count.reserve(sb);
            P.idx.reserve(ni);
            pot_select_count<<<sb, SEL_NT, 0, st>>>(n, P.order.perm.ptr, i0, ni, P.count.ptr);
            pot_select<<<sb, SEL_NT, 0, st>>>(n, P.order.perm.ptr, i0, ni, P.count.ptr, P.idx.ptr);
            NB6_CUDA_CHECK(cudaGetLastError());
            a.idx = P.idx.ptr;
        }
    } else {
        pot_tiles<false><<<P.ntile, JT, 0, st>>>(n, nullptr, P.dm, P.dx, P.keep, P.tiles.ptr, nullptr, a.status,
                                                 P.span.ptr);
        NB6_CUDA_CHECK(cudaGetLastError());
    }
    // two i per thread from a tile of 256 i per eight SMs (the slices fill the
    // rest).  The line matters little: 33.8 us with one and 34.4 with two for a
    // set of 5,000, 108.7 and 106.0 for 12,000, 251 and 245 for 20,000; 4,500 i of
    // 131,071 ordered bodies 368 and 358, 7,000 539 and 559, all of 100,000 3,144
    // and 3,091, of 249,036 18.0 and 17.3 ms; below it 3,000 of 131,071 259 and
    // 272, of 249,036 463 and 450
    const bool two = ni >= 2 * NT * nb6_num_sms() / 8;
    if (ord) two ? pot_launch<2, true>(a, st) : pot_launch<1, true>(a, st);
    else two ? pot_launch<2, false>(a, st) : pot_launch<1, false>(a, st);
    // ordered results are scattered eight bytes at a time: into device memory
    const bool direct = hout && !ord;
    P.out.reserve(ni);
    pot_finalize<<<(ni + 127) / 128, 128, 0, st>>>(P.part.ptr, a.nslices, i0, ni, a.idx,
                                                   direct ? hout : P.out.ptr, a.status,
                                                   direct ? nb6_status_post() : nullptr, ord ? nullptr : P.span.ptr);
    NB6_CUDA_CHECK(cudaGetLastError());
    return direct;
}

void pot_timing_init(cudaStream_t st) {
    if (P.ev0) return;
    NB6_CUDA_CHECK(cudaEventCreate(&P.ev0));
    NB6_CUDA_CHECK(cudaEventCreate(&P.ev1));
    P.span.reserve(1);
    NB6_CUDA_CHECK(cudaMemsetAsync(P.span.ptr, 0, sizeof(DevSpan), st));
}

// The bodies of a call where kernels read them: on the device, or (a small
// host call, which never orders its set) in the pinned staging.
void pot_upload(int n, const double *m, const double *x, cudaStream_t st, bool from_host) {
    P.n = n;
    P.ntile = std::max(1, (n + JT - 1) / JT);
    P.dm = m;
    P.dx = x;
    P.keep = nullptr;
    if (from_host) {
        const size_t np = (size_t)P.ntile * JT, bytes = 4 * np * sizeof(double);
        const Nb6Seg seg[2] = {{0, m, sizeof(double) * n}, {sizeof(double) * np, x, 3 * sizeof(double) * n}};
        P.mx.reserve(4 * np);
        P.dm = static_cast<const double *>(nb6_stage(seg, 2, bytes));
        if (P.dm) {
            P.keep = P.mx.ptr + np;
        } else {
            nb6_upload(P.mx.ptr, seg, 2, bytes, st);
            P.dm = P.mx.ptr;
        }
        P.dx = P.dm + np;
    }
}

}  // namespace

extern "C" {

void gpupot_(int *irank, int *istart, int *ni_, int *n_, double *m, double (*x)[3], double *pot) {
    nb6_devinit_once(irank ? *irank : 0);
    const int n = *n_, ni = *ni_, i0 = *istart - 1;
    if (n <= 0 || ni <= 0 || i0 < 0 || i0 + ni > n) {
        fprintf(stderr, "gpupot: bad range istart=%d ni=%d n=%d\n", *istart, ni, n);
        nb6_fatal(NB6_ERR_BAD_ARG);
        return;
    }
    const double t0 = nb6_wtime();
    cudaStream_t st = nb6_stream();
    pot_timing_init(st);
    P.hout.reserve(ni);
    pot_upload(n, m, &x[0][0], st, true);
    P.stamped = !pot_ordered(ni);
    if (!P.stamped) NB6_CUDA_CHECK(cudaEventRecord(P.ev0, st));
    const bool direct = pot_compute(i0, ni, nb6_uva() ? P.hout.ptr : nullptr, st);
    if (!P.stamped) NB6_CUDA_CHECK(cudaEventRecord(P.ev1, st));
    if (!direct) {
        NB6_CUDA_CHECK(cudaMemcpyAsync(P.hout.ptr, P.out.ptr, sizeof(double) * ni, cudaMemcpyDeviceToHost, st));
        nb6_status_fetch(st);
    }
    NB6_CUDA_CHECK(cudaStreamSynchronize(st));
    if (nb6_check_dev_status() != 0) return;
    memcpy(pot, P.hout.ptr, sizeof(double) * ni);
    if (getenv("NB6_VERBOSE"))
        fprintf(stderr, "[R.%d GPU Pot.A] Ni %d  NTOT %d  pot(s) %f\n", irank ? *irank : 0, ni, n,
                nb6_wtime() - t0);
}

// Extension (no reference counterpart): potential on DEVICE arrays m[n],
// x[n][3]; the result stays on the device, its pointer is returned in *d_out.
// Enqueued on the library stream without a sync.
void nb6_pot_device_(int *istart, int *ni, int *n, const double *d_m, const double *d_x,
                     double **d_out) {
    nb6_devinit_once(0);
    cudaStream_t st = nb6_stream();
    pot_timing_init(st);
    pot_upload(*n, d_m, d_x, st, false);
    P.stamped = !pot_ordered(*ni);
    if (!P.stamped) NB6_CUDA_CHECK(cudaEventRecord(P.ev0, st));
    pot_compute(*istart - 1, *ni, nullptr, st);
    if (!P.stamped) NB6_CUDA_CHECK(cudaEventRecord(P.ev1, st));
    *d_out = P.out.ptr;
}

// Device time (ms) of the last potential call after its upload: packing,
// spatial order, kernel and sums (after a sync).
float nb6_pot_last_kernel_ms_() {
    if (P.stamped) return P.last_ms = nb6_span_ms(P.span.ptr, nb6_stream());
    NB6_CUDA_CHECK(cudaEventSynchronize(P.ev1));
    NB6_CUDA_CHECK(cudaEventElapsedTime(&P.last_ms, P.ev0, P.ev1));
    return P.last_ms;
}

}  // extern "C"
