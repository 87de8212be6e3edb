// Class-tiled H.V (S = 1/2, full basis, R interleaved vectors): the kernel, its
// launchers and the tile sets built per model and R.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <vector>

#include "device.cuh"

namespace pned {

// One class member: acc[j] += c_j w[j ^ D] for the thread's 8 states, with the J
// bits flipped (D) and the J bits that the coefficient depends on (M) fixed by the
// variant (kXVarD, kXVarM).  The jump to the variant is one indexed branch: written
// as a C++ switch it compiles to a tree of compares, about ten branches a member,
// which cost as many issue slots as the products.  `ct` is the shared-memory
// address of the member's table at the thread's hash 0, `h` its hash, `ts` the bytes
// between table entries.  Operands: %0-%15 acc (x, y), %16-%31 w, %32 ct, %33 h, %34 ts, %35 variant.
#define PNED_XA0 "%0", "%1"
#define PNED_XA1 "%2", "%3"
#define PNED_XA2 "%4", "%5"
#define PNED_XA3 "%6", "%7"
#define PNED_XA4 "%8", "%9"
#define PNED_XA5 "%10", "%11"
#define PNED_XA6 "%12", "%13"
#define PNED_XA7 "%14", "%15"
#define PNED_XW0 "%16", "%17"
#define PNED_XW1 "%18", "%19"
#define PNED_XW2 "%20", "%21"
#define PNED_XW3 "%22", "%23"
#define PNED_XW4 "%24", "%25"
#define PNED_XW5 "%26", "%27"
#define PNED_XW6 "%28", "%29"
#define PNED_XW7 "%30", "%31"
// table values n of 2^NB into (x_n, y_n): address ct + (h << NB) * ts, ts apart
#define PNED_XPTR(NB) "shl.b32 t, %33, " #NB "; mad.lo.u32 p, t, %34, %32;\n"
#define PNED_XLC(n) "ld.shared.v2.f64 {x" #n ", y" #n "}, [p]; neg.f64 z" #n ", y" #n "; add.u32 p, p, %34;\n"
#define PNED_XLR(n) "ld.shared.f64 x" #n ", [p]; add.u32 p, p, %34;\n"
#define PNED_XFC_(ax, ay, c, wx, wy)                                                           \
    "fma.rn.f64 " ax ", x" #c ", " wx ", " ax "; fma.rn.f64 " ay ", x" #c ", " wy ", " ay ";\n" \
    "fma.rn.f64 " ax ", z" #c ", " wy ", " ax "; fma.rn.f64 " ay ", y" #c ", " wx ", " ay ";\n"
#define PNED_XFR_(ax, ay, c, wx, wy) \
    "fma.rn.f64 " ax ", x" #c ", " wx ", " ax "; fma.rn.f64 " ay ", x" #c ", " wy ", " ay ";\n"
#define PNED_XFC(A, c, W) PNED_XFC_X(A, c, W)
#define PNED_XFC_X(ax, ay, c, wx, wy) PNED_XFC_(ax, ay, c, wx, wy)
#define PNED_XFR(A, c, W) PNED_XFR_X(A, c, W)
#define PNED_XFR_X(ax, ay, c, wx, wy) PNED_XFR_(ax, ay, c, wx, wy)
// the 8 states' coefficients (c0 .. c7) and partners (w0 .. w7) of a variant
#define PNED_XROWS(F, c0, c1, c2, c3, c4, c5, c6, c7, w0, w1, w2, w3, w4, w5, w6, w7)                                  \
    F(PNED_XA0, c0, PNED_XW##w0) F(PNED_XA1, c1, PNED_XW##w1) F(PNED_XA2, c2, PNED_XW##w2) F(PNED_XA3, c3, PNED_XW##w3) \
    F(PNED_XA4, c4, PNED_XW##w4) F(PNED_XA5, c5, PNED_XW##w5) F(PNED_XA6, c6, PNED_XW##w6) F(PNED_XA7, c7, PNED_XW##w7) \
    "bra DONE;\n"
#define PNED_XL1(L) L(0)
#define PNED_XL2(L) L(0) L(1)
#define PNED_XL4(L) L(0) L(1) L(2) L(3)
#define PNED_XL8(L) L(0) L(1) L(2) L(3) L(4) L(5) L(6) L(7)
// all variants with labels P0 .. P14, products F and table reads L
#define PNED_XALL(P, F, L) \
    P "0:\n" PNED_XPTR(0) PNED_XL1(L) PNED_XROWS(F, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "1:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 1, 0, 1, 0, 1, 0, 1, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "2:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 0, 1, 1, 0, 0, 1, 1, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "3:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 0, 0, 0, 1, 1, 1, 1, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "4:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 1, 2, 3, 0, 1, 2, 3, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "5:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 1, 0, 1, 2, 3, 2, 3, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "6:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 0, 1, 1, 2, 2, 3, 3, 0, 1, 2, 3, 4, 5, 6, 7)    \
    P "7:\n" P "14:\n" PNED_XPTR(3) PNED_XL8(L) PNED_XROWS(F, 0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3, 4, 5, 6, 7) \
    P "8:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 1, 0, 1, 0, 1, 0, 1, 1, 0, 3, 2, 5, 4, 7, 6)    \
    P "9:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 0, 1, 1, 0, 0, 1, 1, 2, 3, 0, 1, 6, 7, 4, 5)    \
    P "10:\n" PNED_XPTR(1) PNED_XL2(L) PNED_XROWS(F, 0, 0, 0, 0, 1, 1, 1, 1, 4, 5, 6, 7, 0, 1, 2, 3)   \
    P "11:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 1, 2, 3, 0, 1, 2, 3, 3, 2, 1, 0, 7, 6, 5, 4)   \
    P "12:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 1, 0, 1, 2, 3, 2, 3, 5, 4, 7, 6, 1, 0, 3, 2)   \
    P "13:\n" PNED_XPTR(2) PNED_XL4(L) PNED_XROWS(F, 0, 0, 1, 1, 2, 2, 3, 3, 6, 7, 4, 5, 2, 3, 0, 1)
#define PNED_XREGS "{\n.reg .f64 x<8>, y<8>, z<8>;\n.reg .u32 t, p;\n"
#define PNED_XTARGETS(P) \
    P "0, " P "1, " P "2, " P "3, " P "4, " P "5, " P "6, " P "7, " P "8, " P "9, " P "10, " P "11, " P "12, " P "13, " P "14"
// real coefficients only, or complex ones with the real members' variants behind them (16 on)
#define PNED_XBODY_R                                                                            \
    PNED_XREGS "TS: .branchtargets " PNED_XTARGETS("V") ";\nbrx.idx.uni %35, TS;\n"             \
    PNED_XALL("V", PNED_XFR, PNED_XLR) "DONE:\n}\n"
#define PNED_XBODY_C                                                                                              \
    PNED_XREGS "TS: .branchtargets " PNED_XTARGETS("V") ", V14, " PNED_XTARGETS("U") ";\nbrx.idx.uni %35, TS;\n"   \
    PNED_XALL("V", PNED_XFC, PNED_XLC) PNED_XALL("U", PNED_XFR, PNED_XLR) "DONE:\n}\n"

template <bool RC>
__device__ __forceinline__ void x_member(const uint4 &S, uint32_t base, uint32_t tab, uint32_t ts,
                                         const double2 (&w)[kXSPT], double2 (&acc)[kXSPT])
{
    static_assert(kXSPT == 8, "the variants below are written for 8 states a thread");
    const uint32_t h = ((base & S.x) * S.y) >> ((S.w >> 8) & 31u), ct = tab + (S.w >> 16) * ts;
    const uint32_t var = (S.w & 15u) | (RC ? 0u : (S.w >> 9) & 16u);   // kXReal: the real variants
#define PNED_XOPS                                                                                                        \
    "+d"(acc[0].x), "+d"(acc[0].y), "+d"(acc[1].x), "+d"(acc[1].y), "+d"(acc[2].x), "+d"(acc[2].y), "+d"(acc[3].x),      \
        "+d"(acc[3].y), "+d"(acc[4].x), "+d"(acc[4].y), "+d"(acc[5].x), "+d"(acc[5].y), "+d"(acc[6].x), "+d"(acc[6].y),  \
        "+d"(acc[7].x), "+d"(acc[7].y)                                                                                   \
        : "d"(w[0].x), "d"(w[0].y), "d"(w[1].x), "d"(w[1].y), "d"(w[2].x), "d"(w[2].y), "d"(w[3].x), "d"(w[3].y),        \
          "d"(w[4].x), "d"(w[4].y), "d"(w[5].x), "d"(w[5].y), "d"(w[6].x), "d"(w[6].y), "d"(w[7].x), "d"(w[7].y),        \
          "r"(ct), "r"(h), "r"(ts), "r"(var)                                                                             \
        : "memory"
    if (RC) asm volatile(PNED_XBODY_R : PNED_XOPS);
    else asm volatile(PNED_XBODY_C : PNED_XOPS);
#undef PNED_XOPS
}

// One pass of the class-tiled kernel.  A block owns tiles of 2048 elements: 2^lr of
// the R vectors (its group ch) times 2^(11 - lr) states; thread t holds vector t mod
// 2^lr of the 8 states of one row (rows on the bits of t above lr, J bits jexp).  The
// own rows come into shared memory by cp.async and the in-tile classes gather there;
// the out-of-tile classes read their partner rows through L1/L2 meanwhile.
//
// What bounds it: not memory (N = 22, R = 16 with a field: DRAM at a third of its
// rate, the L1 data path 50-58 % busy) but instructions and their latency at 16 warps per
// SM: fp64 pipe 25 %, issue 48 %.  Hence the classes (60 masks become 40 row reads at
// N = 24), the perfect hash (3 instructions for a coefficient index), members as one
// 16-byte constant read fetched ahead, and the indexed jump.  Measured H.V against the
// multi-vector kernel: N = 24, R = 16 with a field 18.6 -> 12.6 ms, R = 12 without
// 11.8 -> 8.1 ms, N = 22, R = 2 with a field 0.675 -> 0.429 ms, N = 26, R = 4 with a field
// 21.5 -> 13.0 ms, without 14.9 -> 9.5 ms.
// Measured and dropped, on an earlier form: a second class in flight through cp.async (15.1
// against 14.8 ms: the address arithmetic costs more than the latency it hides).
template <bool RC, bool RD, int K, bool SLOT>
__global__ void __launch_bounds__(kThreads, 2)
    hv_xtile_kernel(const __grid_constant__ XTileProgram prog, const HvArgs a, int nch)
{
    // 128-byte aligned: a warp's rows then fill whole shared-memory lines.  Without it the static
    // arrays in front decide (H.V with four sums, N = 22, R = 16 with a field: 3.55 ms 16 bytes off a
    // line, 3.46 ms 32 bytes off, 3.42 ms aligned; N = 20, R = 6: 0.371, 0.350, 0.350)
    extern __shared__ __align__(128) double2 smem[];
    const uint32_t tid = threadIdx.x;
    const int lr = prog.lr, rc = 1 << lr, R = a.R;
    const int ch = int(blockIdx.x) % nch;            // the block's group of vectors
    const int r = int(tid) & (rc - 1), rg = ch * rc + r;   // vector in the group and in the batch
    double2 *s_v = smem;
    double2 *s_pw = smem + kXTile;
    double *s_d = reinterpret_cast<double *>(s_pw + kXTile);   // real diagonal: per state (SLOT: per element)
    double2 *s_tab = reinterpret_cast<double2 *>(s_d + (RD ? kXTile : 0));
    if (SLOT) {
        for (int i = tid; i < prog.ntab * rc; i += kThreads) {
            const int src = prog.tsrc[i >> lr];
            s_tab[i] = src == 0xffff ? make_double2(0.0, 0.0) : a.table[src * R + ch * rc + (i & (rc - 1))];
        }
    } else {
        for (int i = tid; i < prog.ntab; i += kThreads) {
            const int src = prog.tsrc[i];
            s_tab[i] = src == 0xffff ? make_double2(0.0, 0.0) : a.table[src];
        }
    }
    const uint32_t tabp = uint32_t(__cvta_generic_to_shared(s_tab + (SLOT ? r : 0))), ts = SLOT ? 16u << lr : 16u;
    const double2 *pw_src = prog.first ? a.P : a.W;
    const double sc = a.sc[rg], pc = a.pc ? a.pc[rg] : 0.0, gs = a.gsc ? a.gsc[rg] : 0.0;
    const double hs = a.hsc ? a.hsc[rg] : sc;
    const double shift = a.shift + (a.shiftv ? a.shiftv[rg] : 0.0);
    const int64_t R16 = int64_t(R) * 16, rg16 = int64_t(rg) * 16;
    const int64_t jo0 = int64_t(prog.jexp[1]) * R16, jo1 = int64_t(prog.jexp[2]) * R16,
                  jo2 = int64_t(prog.jexp[4]) * R16;   // byte offsets of the J bits
    auto at = [&](const double2 *p, int64_t off, int j) {   // the thread's j-th state of a row at byte offset off
        return reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(p) + off + ((j & 1) ? jo0 : 0) +
                                                 ((j & 2) ? jo1 : 0) + ((j & 4) ? jo2 : 0));
    };
    // requests the epilogue's rows of P or W and the diagonal into the thread's own slots
    auto epilogue_rows = [&](uint32_t base, int64_t off) {
        if (pw_src) {
#pragma unroll
            for (int j = 0; j < kXSPT; ++j) cp_async16(s_pw + tid + kThreads * j, at(pw_src, off, j));
        }
        if (RD && prog.first) {
            // the thread's own diagonal values (lanes of one state copy the same value)
#pragma unroll
            for (int j = 0; j < kXSPT; ++j) {
                const int64_t st = int64_t(base | prog.jexp[j]);
                cp_async8(s_d + tid + kThreads * j,
                          static_cast<const double *>(a.diag) + (SLOT ? st * R + rg : st));
            }
        }
        cp_async_commit();
    };
    double2 red[K];
#pragma unroll
    for (int k = 0; k < K; ++k) red[k] = make_double2(0.0, 0.0);
    uint32_t rowbase = 0;
    for (int k = 0; k < prog.rbits; ++k) rowbase |= ((tid >> (lr + k)) & 1u) << prog.rowpos[k];
    const int64_t ntiles = int64_t(1) << prog.nouter;
    __shared__ uint32_t s_next;
    __shared__ double2 s_red[kThreads / 32][K][kXMaxVec];
    uint32_t *const ctr = a.tile_counter ? a.tile_counter + prog.pass * nch + ch : nullptr;
    const int64_t ct = ctr ? int64_t(max(1, a.rv_chunk)) : 1;
    const int64_t nchunks = (ntiles + ct - 1) / ct;
    const int64_t blk = int64_t(blockIdx.x) / nch, nblk = int64_t(gridDim.x) / nch;
    int64_t chunk = blk;
    if (ctr) {
        if (tid == 0) s_next = atomicAdd(ctr, 1u);
        __syncthreads();
        chunk = s_next;
    }
    while (chunk < (ctr ? nchunks : ntiles)) {
        const int64_t tile_end = ctr ? min(ntiles, (chunk + 1) * ct) : chunk + 1;
        for (int64_t tile = ctr ? chunk * ct : chunk; tile < tile_end; ++tile) {
            uint32_t base = rowbase;
            for (int k = 0; k < prog.nouter; ++k) base |= uint32_t((tile >> k) & 1) << prog.outer[k];
            __syncthreads();   // the previous tile's shared reads are done (first tile: table staged)
            if (ctr && tid == 0 && tile == chunk * ct) s_next = atomicAdd(ctr, 1u);   // all have read s_next
            const int64_t off = int64_t(base) * R16 + rg16;
#pragma unroll
            for (int j = 0; j < kXSPT; ++j) cp_async16(s_v + tid + kThreads * j, at(a.C, off, j));
            cp_async_commit();
            epilogue_rows(base, off);
            double2 acc[kXSPT];
#pragma unroll
            for (int j = 0; j < kXSPT; ++j) acc[j] = make_double2(0.0, 0.0);
            // out-of-tile classes through L1/L2 while the own rows land, then the in-tile ones
            uint4 nx = prog.s[0];
            double2 w[kXSPT];
#pragma unroll 1
            for (int m = 0; m < prog.nsub; ++m) {
                const uint4 S = nx;
                nx = prog.s[m + 1];
                if (S.w & 128u) {   // a new class: its partner rows
                    const uint32_t dg = (S.w & 15u) == uint32_t(kXGeneric) ? (S.w >> 4) & 7u : 0u;
                    if (m < prog.nout) {
                        if (dg == 0) {
                            const int64_t po = int64_t(base ^ S.z) * R16 + rg16;
#pragma unroll
                            for (int j = 0; j < kXSPT; ++j) w[j] = __ldg(at(a.C, po, j));
                        } else {
#pragma unroll
                            for (int j = 0; j < kXSPT; ++j)
                                w[j] = __ldg(a.C + (int64_t(base ^ S.z ^ prog.jexp[uint32_t(j) ^ dg]) * R + rg));
                        }
                    } else {
                        if (m == prog.nout) {   // the first in-tile class
                            cp_async_wait<1>();
                            __syncthreads();
                        }
                        const double2 *sv = s_v + (tid ^ (S.z << lr));
                        if (dg == 0) {
#pragma unroll
                            for (int j = 0; j < kXSPT; ++j) w[j] = sv[kThreads * j];
                        } else {
#pragma unroll
                            for (int j = 0; j < kXSPT; ++j) w[j] = sv[kThreads * (uint32_t(j) ^ dg)];
                        }
                    }
                }
                x_member<RC>(S, base, tabp, ts, w, acc);
            }
            cp_async_wait<0>();
            double2 g[K >= 4 ? kXSPT : 1];
            if (K >= 4 && prog.last && a.G) {
#pragma unroll
                for (int j = 0; j < kXSPT; ++j) g[j] = __ldcs(at(a.G, off, j));
            }
#pragma unroll
            for (int j = 0; j < kXSPT; ++j) {
                const int sl = int(tid) + kThreads * j;
                const double2 v = s_v[sl];
                double2 hsum = acc[j];
                if (prog.first) {
                    if (RD) {
                        const double dd = s_d[sl] - shift;
                        hsum.x = fma(dd, v.x, hsum.x);
                        hsum.y = fma(dd, v.y, hsum.y);
                    } else {
                        double2 dd = __ldcs(static_cast<const double2 *>(a.diag) + int64_t(base | prog.jexp[j]));
                        dd.x -= shift;
                        hsum = cfma(dd, v, hsum);
                    }
                }
                const double2 hv = cscale(hs, hsum);
                double2 o = hv;
                if (!prog.first) {
                    const double2 w0 = s_pw[sl];
                    o.x += w0.x;
                    o.y += w0.y;
                } else if (a.P) {
                    const double2 p = s_pw[sl];
                    o.x = fma(pc, p.x, o.x);
                    o.y = fma(pc, p.y, o.y);
                }
                __stcs(const_cast<double2 *>(at(a.W, off, j)), o);
                red[0].x = fma(v.x, hsum.x, fma(v.y, hsum.y, red[0].x));
                red[0].y = fma(v.x, hsum.y, fma(-v.y, hsum.x, red[0].y));
                if (!prog.last) continue;
                const double2 vv = cscale(sc, v);
                if (K >= 2) red[1].x += o.x * o.x + o.y * o.y;
                if (K >= 4 && a.G) {
                    const double2 gv = cscale(gs, g[j]);
                    red[2] = cadd(red[2], cconjmul(gv, o));
                    red[3] = cadd(red[3], cconjmul(gv, vv));
                }
            }
        }
        if (!ctr) {
            chunk += nblk;
            continue;
        }
        red[0] = cscale(sc * hs, red[0]);   // <v|Hv> was summed unscaled
        x_sums_store<K>(red, s_red, lr, R, ch, a.partials + size_t(chunk) * K * R);
        chunk = s_next;
    }
    if (!ctr) red[0] = cscale(sc * hs, red[0]);
    if (!ctr) x_sums_store<K>(red, s_red, lr, R, ch, a.partials + size_t(blk) * K * R);
    if (K == 1 && prog.last) hv_finish(a, smem);   // the tile buffer is free behind the first barrier in there
}

const pned_model::XTileSet *find_xtiles(const pned_model *m, int R)
{
    std::lock_guard<std::mutex> lock(const_cast<pned_model *>(m)->rtiles_mu);
    auto it = m->xtiles.find(R);
    if (it == m->xtiles.end() || it->second.off || it->second.progs.empty()) return nullptr;
    return &it->second;
}

static size_t xtile_smem(const pned_model *m, const pned_model::XTileSet &xs, bool slot_tables)
{
    int ntab = 1;
    for (const auto &t : xs.progs) ntab = std::max(ntab, t->ntab);
    return sizeof(double2) * (2 * size_t(kXTile) + size_t(ntab) * (slot_tables ? (1 << xs.lr) : 1)) +
           (m->real_diag ? sizeof(double) * kXTile : 0);
}

bool ensure_xtiles(pned_model *m, int R, bool slot_tables)
{
    const HostProgram &hp = m->hp;
    if (pick_vpt(R) == 0) return false;
    // One vector: only for complex coefficients (Gamma, a field, slot couplings) -- with real
    // ones a member is half the products, and the tensor-copy kernel is faster -- and only from
    // 26 sites on (N = 26: 3.88 -> 3.21 ms, N = 28: 16.1 -> 14.0 ms).  Smaller bases keep the
    // gather kernel's order of additions although it is slower (N = 24: 0.98 against 0.82 ms):
    // the sign of the Ritz vector that vec12 finds turns on the last bit of alpha and beta, so
    // another order may return -x where a caller had x.
    if (R == 1 && (m->real_coef || hp.n < kTileBigSites)) return false;
    // Slot tables are staged per vector of the group, so a call needs more tiles to pay: 2^19
    // elements (step of 4 slots: N = 16 52.8 against 51.2 us with the multi-vector kernel, N = 18
    // 98.5 against 114.6), and for 6 slots, groups of two, 2^22 (N = 18 189 against 159 us, N = 20
    // 543 against 642).
    if (slot_tables && double(hp.dim) * R < double(R == 6 ? 1 << 22 : 1 << 19)) return false;
    std::lock_guard<std::mutex> lock(m->rtiles_mu);
    pned_model::XTileSet &xs = m->xtiles[R];
    if (xs.off || xs.built) return !xs.off && !xs.progs.empty();
    xs.built = true;
    std::vector<XTilePass> ps;
    if (plan_xtiles_for(hp, R, xs.lr, ps) != PNED_OK) return false;
    std::vector<uint16_t> tsrc;   // of all passes
    for (size_t p = 0; p < ps.size(); ++p) {
        const XTilePass &t = ps[p];
        if (t.subs.size() > size_t(kMaxTerms)) { xs.progs.clear(); return false; }
        std::unique_ptr<XTileProgram> T(new XTileProgram());
        T->lr = xs.lr;
        T->rbits = int(t.rowpos.size());
        T->nsub = int(t.subs.size());
        T->nout = t.nout;
        T->ntab = int(t.tsrc.size());
        for (int x : t.tsrc) tsrc.push_back(uint16_t(x < 0 ? 0xffff : x));
        T->nouter = int(t.outer.size());
        T->first = p == 0;
        T->last = p + 1 == ps.size();
        T->pass = int(p);
        for (int j = 0; j < kXSPT; ++j)
            for (int k = 0; k < kXJB; ++k)
                if ((j >> k) & 1) T->jexp[j] |= 1u << t.jpos[k];
        for (int k = 0; k < T->rbits; ++k) T->rowpos[k] = uint8_t(t.rowpos[k]);
        for (int k = 0; k < T->nouter; ++k) T->outer[k] = uint8_t(t.outer[k]);
        for (size_t i = 0; i < t.subs.size(); ++i) {
            const XSub &q = t.subs[i];
            T->s[i] = make_uint4(q.dmask, q.mul, q.mask, m->table_varies ? q.pack & ~kXReal : q.pack);
        }
        xs.groups += t.groups;
        xs.progs.push_back(std::move(T));
    }
    if (!xs.mem.upload(tsrc.data(), sizeof(uint16_t) * tsrc.size())) {   // no room now: the next context asks again
        xs.progs.clear();
        xs.groups = 0;
        xs.built = false;
        return false;
    }
    const uint16_t *src = static_cast<const uint16_t *>(xs.mem.p);
    for (auto &T : xs.progs) {
        T->tsrc = src;
        src += T->ntab;
    }
    // two blocks' shared memory per SM
    if (2 * (xtile_smem(m, xs, slot_tables) + 5 * 1024) > 227 * 1024) { xs.progs.clear(); return false; }
    return true;
}

void switch_xtiles(pned_model *m, int R, bool on)
{
    std::lock_guard<std::mutex> lock(m->rtiles_mu);
    m->xtiles[R].off = !on;
}

static int xtile_grid(const pned_model *m, const pned_model::XTileSet &xs, int R, int nblocks)
{
    const int nch = R >> xs.lr;
    return std::max(1, std::min(nblocks, 2 * m->nsm) / nch) * nch;
}

// Tiles per chunk in the dynamic order (one partial-sum record each): up to four, but
// at least eight chunks a block, so that the last ones spread over the device.
static int64_t xtile_chunk(const XTileProgram &t, int per_ch)
{
    return std::max<int64_t>(1, std::min<int64_t>(4, (int64_t(1) << t.nouter) / (8 * int64_t(per_ch))));
}
static int64_t xtile_chunks(const XTileProgram &t, int per_ch)
{
    const int64_t c = xtile_chunk(t, per_ch);
    return ((int64_t(1) << t.nouter) + c - 1) / c;
}

int64_t xtile_rows(const pned_model *m, const pned_model::XTileSet &xs, int R, int nblocks, bool dynamic)
{
    const int per = xtile_grid(m, xs, R, nblocks) / (R >> xs.lr);
    int64_t n = 0;
    for (const auto &t : xs.progs) n += dynamic ? xtile_chunks(*t, per) : per;
    return n;
}

template <bool RC, bool RD, int K, bool SLOT>
static cudaError_t launch_xtile_t(const pned_model *m, const pned_model::XTileSet &xs, const HvArgs &a, int nblocks,
                                  cudaStream_t st)
{
    auto kern = hv_xtile_kernel<RC, RD, K, SLOT>;
    const size_t smem = xtile_smem(m, xs, SLOT);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kern), m->device);
    if (e == cudaSuccess && m->carveout) e = set_carveout(reinterpret_cast<const void *>(kern), m->device, smem, 2);
    if (e != cudaSuccess) return e;
    const int nch = a.R >> xs.lr, grid = xtile_grid(m, xs, a.R, nblocks), per = grid / nch;
    const bool dyn = tile_dynamic(m, a, nblocks);
    HvArgs b = a;
    if (!dyn) b.tile_counter = nullptr;
    else if (!a.fin.out &&
             (e = cudaMemsetAsync(a.tile_counter, 0, sizeof(uint32_t) * xs.progs.size() * nch, st)) != cudaSuccess)
        return e;
    size_t off = 0;
    for (size_t p = 0; p < xs.progs.size(); ++p) {
        b.partials = a.partials + off;
        b.rv_chunk = int(xtile_chunk(*xs.progs[p], per));
        off += (dyn ? size_t(xtile_chunks(*xs.progs[p], per)) : size_t(per)) * K * a.R;
        kern<<<grid, kThreads, smem, st>>>(*xs.progs[p], b, nch);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int K>
static cudaError_t launch_xtile_k(const pned_model *m, const pned_model::XTileSet &xs, const HvArgs &a, int nblocks,
                                  cudaStream_t st)
{
    if (a.slot_tables) return launch_xtile_t<false, true, K, true>(m, xs, a, nblocks, st);
    if (m->real_coef && m->real_diag) return launch_xtile_t<true, true, K, false>(m, xs, a, nblocks, st);
    if (m->real_diag) return launch_xtile_t<false, true, K, false>(m, xs, a, nblocks, st);
    return launch_xtile_t<false, false, K, false>(m, xs, a, nblocks, st);
}

cudaError_t launch_xtile(const pned_model *m, const pned_model::XTileSet &xs, const HvArgs &a, int nblocks,
                         cudaStream_t st)
{
    if (a.K == 1) return launch_xtile_k<1>(m, xs, a, nblocks, st);
    if (a.K == 4) return launch_xtile_k<4>(m, xs, a, nblocks, st);
    return cudaErrorInvalidValue;
}

}   // namespace pned
