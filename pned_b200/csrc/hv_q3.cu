// Tiled S = 1 H.v (base 3, full basis, one vector): the kernel, its launcher and the tile
// sets built per model.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <vector>

#include "device.cuh"

namespace pned {

constexpr int kQ3States = 9;       // states a thread: the digits of the two J sites
constexpr int kQ3Threads = 256;    // threads a block at most

// acc[ja, jb] += c w[ja + DA, jb + DB] over the rows that stay in 0..2.  M: the J digits
// that the coefficient depends on (1: ja, 2: jb, 3: both); ct points at its values.
template <int DA, int DB, int M, bool RC>
__device__ __forceinline__ void q3_apply(const double2 *ct, const double2 (&w)[kQ3States], double2 (&acc)[kQ3States])
{
#pragma unroll
    for (int jb = 0; jb < 3; ++jb)
#pragma unroll
        for (int ja = 0; ja < 3; ++ja) {
            if (ja + DA < 0 || ja + DA > 2 || jb + DB < 0 || jb + DB > 2) continue;
            const int ci = (M & 1 ? ja : 0) + (M == 3 ? 3 * jb : (M == 2 ? jb : 0));
            const int j = ja + 3 * jb, jw = j + DA + 3 * DB;
            if (RC) {
                const double c = ct[ci].x;
                acc[j].x = fma(c, w[jw].x, acc[j].x);
                acc[j].y = fma(c, w[jw].y, acc[j].y);
            } else {
                acc[j] = cfma(ct[ci], w[jw], acc[j]);
            }
        }
}

// One pass: a tile is the 3^k states of k sites; thread t owns the 9 states of the two J
// sites (local digits 0 and 1) for one setting of the others.  Members with
// the same offset outside J share their nine partner rows (a class, as in hv_xtile.cu), and
// their J part is a fixed register shift, so a term costs one row read and two products a
// state; the kernel for any base (hv_qtile.cu) reads a coefficient and decodes the pair
// state for every state and term as well.
//
// What bounds it: instructions and shared-memory reads, not memory (N = 16: 3.66 ms for 5
// passes that move 10 GB).  H.v of one vector: N = 18 50.2 -> 32.3 ms, N = 16 5.57 -> 3.66 ms,
// N = 14 with a field 1.20 -> 0.66 ms; Lanczos step N = 12 0.113 -> 0.080 ms.  Rows and the epilogue's
// P or W and diagonal come in by cp.async in global order; local slots are nine apart from
// lane to lane, so the 16-byte reads have no bank conflicts.
template <bool RC, bool RD, int K>
__global__ void __launch_bounds__(kQ3Threads, 2) hv_q3_kernel(const __grid_constant__ Q3Program prog, const HvArgs a)
{
    extern __shared__ double2 smem[];
    const int nt = prog.nt, nth = int(blockDim.x), tid = int(threadIdx.x);
    double2 *s_v = smem;                           // [nt]
    double2 *s_pw = s_v + nt;                      // rows of P or W, laid out as s_v
    double2 *s_tab = s_pw + nt;
    double *s_d = reinterpret_cast<double *>(s_tab + prog.ntab);             // [nt] real diagonal (first pass)
    uint32_t *s_goff = reinterpret_cast<uint32_t *>(s_d + (RD ? nt : 0));    // [nt] global offset of local slot
    uint16_t *s_slot = reinterpret_cast<uint16_t *>(s_goff + nt);            // [nt] local slot in global order
    for (int i = tid; i < prog.ntab; i += nth) s_tab[i] = prog.tab[i];
    for (int l = tid; l < nt; l += nth) {
        uint32_t off = 0, rank = 0;
        int x = l;
        for (int i = 0; i < prog.k; ++i) {
            const int d = x % 3;
            x /= 3;
            off += uint32_t(d) * prog.spow[i];
            rank += uint32_t(d) * prog.rank[i];
        }
        s_goff[l] = off;
        s_slot[rank] = uint16_t(l);
    }
    double2 red[K];
#pragma unroll
    for (int k = 0; k < K; ++k) red[k] = make_double2(0.0, 0.0);
    const int nitems = nt / kQ3States;   // item t: the states 9 t .. 9 t + 8
    const double sc = a.sc[0], pc = a.pc ? a.pc[0] : 0.0, gs = a.gsc ? a.gsc[0] : 0.0;
    const double2 *pw_src = prog.first ? a.P : a.W;
    __shared__ uint32_t s_base;
    for (int64_t tile = blockIdx.x; tile < prog.ntiles; tile += gridDim.x) {
        __syncthreads();   // the previous tile's shared reads are done (first tile: tables staged)
        if (tid == 0) {
            uint32_t b = 0, x = uint32_t(tile);
            for (int i = 0; i < prog.nouter; ++i) {
                const uint32_t y = x / 3u;
                b += (x - 3u * y) * prog.opow[i];
                x = y;
            }
            s_base = b;
        }
        __syncthreads();
        const uint32_t base = s_base;
        for (int i = tid; i < nt; i += nth) {
            const int l = s_slot[i];
            cp_async16(s_v + l, a.C + (base + s_goff[l]));
        }
        cp_async_commit();
        if (pw_src)
            for (int i = tid; i < nt; i += nth) {
                const int l = s_slot[i];
                cp_async16(s_pw + l, pw_src + (base + s_goff[l]));
            }
        if (RD && prog.first)
            for (int i = tid; i < nt; i += nth) {
                const int l = s_slot[i];
                cp_async8(s_d + l, static_cast<const double *>(a.diag) + (base + s_goff[l]));
            }
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        bool landed = false;   // the epilogue's rows
        for (int it = tid; it < nitems || !landed; it += nth) {
            const bool on = it < nitems;
            const int t9 = on ? it * kQ3States : 0;
            uint32_t dig = 0;   // the other digits, 2 bits each (digit 2 + i at bits 2 i)
            {
                int x = t9 / kQ3States;
                for (int i = 0; i < prog.k - 2; ++i) {
                    const int y = x / 3;
                    dig |= uint32_t(x - 3 * y) << (2 * i);
                    x = y;
                }
            }
            double2 acc[kQ3States], w[kQ3States];
#pragma unroll
            for (int j = 0; j < kQ3States; ++j) acc[j] = make_double2(0.0, 0.0);
            for (int m = 0; m < prog.nsub; ++m) {
                const Q3Sub S = prog.s[m];
                if (S.first) {
                    // an offset that leaves the tile belongs to zero coefficients: clamped
                    const double2 *p = s_v + min(max(t9 + S.loff, 0), nt - kQ3States);
#pragma unroll
                    for (int j = 0; j < kQ3States; ++j) w[j] = p[j];
                }
                const double2 *ct = s_tab + S.tab + ((dig >> S.sh1) & 3u) * S.m1 + ((dig >> S.sh2) & 3u) * S.m2;
                switch (S.var) {
                case 0: q3_apply<0, 0, 0, RC>(ct, w, acc); break;
                case 1: q3_apply<-1, 0, 1, RC>(ct, w, acc); break;
                case 2: q3_apply<0, 0, 1, RC>(ct, w, acc); break;
                case 3: q3_apply<1, 0, 1, RC>(ct, w, acc); break;
                case 4: q3_apply<0, -1, 2, RC>(ct, w, acc); break;
                case 5: q3_apply<0, 0, 2, RC>(ct, w, acc); break;
                case 6: q3_apply<0, 1, 2, RC>(ct, w, acc); break;
                case 7: q3_apply<-1, -1, 3, RC>(ct, w, acc); break;
                case 8: q3_apply<0, -1, 3, RC>(ct, w, acc); break;
                case 9: q3_apply<1, -1, 3, RC>(ct, w, acc); break;
                case 10: q3_apply<-1, 0, 3, RC>(ct, w, acc); break;
                case 11: q3_apply<1, 0, 3, RC>(ct, w, acc); break;
                case 12: q3_apply<-1, 1, 3, RC>(ct, w, acc); break;
                case 13: q3_apply<0, 1, 3, RC>(ct, w, acc); break;
                default: q3_apply<1, 1, 3, RC>(ct, w, acc); break;
                }
            }
            if (!landed) {
                cp_async_wait<0>();
                __syncthreads();
                landed = true;
            }
            if (!on) continue;
            double2 g[K >= 4 ? kQ3States : 1];
            if (K >= 4 && prog.last && a.G) {
#pragma unroll
                for (int j = 0; j < kQ3States; ++j) g[j] = __ldcs(a.G + (base + s_goff[t9 + j]));
            }
#pragma unroll
            for (int j = 0; j < kQ3States; ++j) {
                const uint32_t st = base + s_goff[t9 + j];
                const double2 v = s_v[t9 + j];
                double2 hsum = acc[j];
                if (prog.first) {
                    if (RD) {
                        const double dd = s_d[t9 + j] - a.shift;
                        hsum.x = fma(dd, v.x, hsum.x);
                        hsum.y = fma(dd, v.y, hsum.y);
                    } else {
                        double2 dd = __ldcs(static_cast<const double2 *>(a.diag) + st);
                        dd.x -= a.shift;
                        hsum = cfma(dd, v, hsum);
                    }
                }
                const double2 hv = cscale(sc, hsum);
                double2 out = hv;
                if (pw_src) {
                    const double2 p = s_pw[t9 + j];
                    const double f = prog.first ? pc : 1.0;
                    out.x = fma(f, p.x, out.x);
                    out.y = fma(f, p.y, out.y);
                }
                __stcs(a.W + st, out);
                const double2 vv = cscale(sc, v);
                red[0] = cadd(red[0], cconjmul(vv, hv));
                if (!prog.last) continue;
                if (K >= 2) red[K >= 2 ? 1 : 0].x += out.x * out.x + out.y * out.y;
                if (K >= 4 && a.G) {
                    const double2 gv = cscale(gs, g[j]);
                    red[K >= 4 ? 2 : 0] = cadd(red[K >= 4 ? 2 : 0], cconjmul(gv, out));
                    red[K >= 4 ? 3 : 0] = cadd(red[K >= 4 ? 3 : 0], cconjmul(gv, vv));
                }
            }
        }
    }
    // block sums in a fixed order
    __syncthreads();
    double2 *sm = s_v;   // [nth][K] (the tile buffer holds more)
#pragma unroll
    for (int k = 0; k < K; ++k) sm[tid * K + k] = red[k];
    __syncthreads();
    for (int w = kQ3Threads / 2; w > 0; w >>= 1) {
        if (w < nth && tid < w && tid + w < nth) {
#pragma unroll
            for (int k = 0; k < K; ++k) sm[tid * K + k] = cadd(sm[tid * K + k], sm[(tid + w) * K + k]);
        }
        __syncthreads();
    }
    if (tid < K) a.partials[size_t(blockIdx.x) * K + tid] = sm[tid];
}

const pned_model::Q3Set *find_q3(const pned_model *m, int R)
{
    std::lock_guard<std::mutex> lock(const_cast<pned_model *>(m)->rtiles_mu);
    auto it = m->q3.find(R);
    if (it == m->q3.end() || it->second.progs.empty()) return nullptr;
    return &it->second;
}

int q3_grid(const pned_model *m, const pned_model::Q3Set &qs, int nblocks)
{
    const int per_sm = std::max<int>(1, std::min<int>(512 / qs.threads, int(227 * 1024 / (qs.smem + 1024))));
    return std::max(1, std::min(nblocks, per_sm * m->nsm));
}

template <bool RC, bool RD, int K>
static cudaError_t launch_q3_t(const pned_model *m, const pned_model::Q3Set &qs, const HvArgs &a, int nblocks,
                               cudaStream_t st)
{
    auto kern = hv_q3_kernel<RC, RD, K>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kern), m->device);
    if (e != cudaSuccess) return e;
    const int grid = q3_grid(m, qs, nblocks);
    HvArgs b = a;
    for (size_t p = 0; p < qs.progs.size(); ++p) {
        b.partials = a.partials + size_t(p) * grid * K;
        kern<<<grid, qs.threads, qs.smem, st>>>(*qs.progs[p], b);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int K>
static cudaError_t launch_q3_k(const pned_model *m, const pned_model::Q3Set &qs, const HvArgs &a, int nblocks,
                               cudaStream_t st)
{
    if (m->real_coef && m->real_diag) return launch_q3_t<true, true, K>(m, qs, a, nblocks, st);
    if (m->real_diag) return launch_q3_t<false, true, K>(m, qs, a, nblocks, st);
    return launch_q3_t<false, false, K>(m, qs, a, nblocks, st);
}

cudaError_t launch_q3(const pned_model *m, const pned_model::Q3Set &qs, const HvArgs &a, int nblocks, cudaStream_t st)
{
    if (a.K == 1) return launch_q3_k<1>(m, qs, a, nblocks, st);
    if (a.K == 4) return launch_q3_k<4>(m, qs, a, nblocks, st);
    return cudaErrorInvalidValue;
}

// The S = 1 passes for one vector (several: the kernel for any base runs, whose threads
// share a term's decode over their vectors; a form of this kernel with all vectors in one
// tile took 21.6 against 20.6 ms a step at N = 16, R = 4, and 0.52 against 0.41 ms at N = 12,
// R = 8): the largest tile whose two buffers, tables and index
// arrays leave room for two blocks per SM.  From 9 sites on: at 8 a tile is 729 states, 81
// items, so nine blocks of three warps run, each thread's nine states one after another
// (Lanczos step 31.1 against 27.2 us with the kernel for any base, mTPQ step 35.9 against
// 25.4 us; N = 9, 243 items: 36.2 against 52.8 and 42.4 against 52.7).  False (any other base,
// an element that moves a digit by two, no room): the kernel for any base runs.
bool ensure_q3(pned_model *m, int R)
{
    const HostProgram &hp = m->hp;
    if (hp.q != 3 || hp.sector || hp.n < 9 || hp.n > 20 || R != 1) return false;
    std::lock_guard<std::mutex> lock(m->rtiles_mu);
    if (m->q3.count(R)) return !m->q3[R].progs.empty();
    pned_model::Q3Set &qs = m->q3[R];
    int64_t pw[32];
    pw[0] = 1;
    for (int i = 1; i <= hp.n; ++i) pw[i] = pw[i - 1] * 3;
    auto smem_of = [&](int k, int ntab) {
        const int nt = int(pw[k]);
        return sizeof(double2) * (2 * size_t(nt) + ntab) + size_t(nt) * (sizeof(double) + 6) + 16;
    };
    int k = 3;
    while (k + 1 <= std::min(hp.n - 2, 7) && smem_of(k + 1, kQ3MaxTab) <= 112 * 1024) ++k;
    if (smem_of(k, kQ3MaxTab) > 112 * 1024) return false;
    std::vector<Q3Pass> passes;
    if (plan_q3(hp, k, 1, passes) != PNED_OK || passes.size() > size_t(kQTileMaxPasses)) return false;
    int ntab = 1;
    for (size_t p = 0; p < passes.size(); ++p) {
        const Q3Pass &ps = passes[p];
        if (ps.subs.size() > size_t(kQ3MaxSubs) || ps.tsrc.size() > size_t(kQ3MaxTab)) { qs.progs.clear(); return false; }
        std::unique_ptr<Q3Program> T(new Q3Program());
        T->k = k;
        T->nt = int(pw[k]);
        T->nouter = int(ps.outer.size());
        T->nsub = int(ps.subs.size());
        T->ntab = int(ps.tsrc.size());
        T->first = p == 0;
        T->last = p + 1 == passes.size();
        T->ntiles = pw[hp.n - k];
        for (int i = 0; i < k; ++i) {
            T->spow[i] = uint32_t(pw[ps.sites[i]]);
            int below = 0;   // tile sites below: the digit's weight in global order
            for (int x : ps.sites) below += x < ps.sites[i];
            T->rank[i] = uint32_t(pw[below]);
        }
        for (int i = 0; i < T->nouter; ++i) T->opow[i] = uint32_t(pw[ps.outer[i]]);
        for (size_t i = 0; i < ps.tsrc.size(); ++i) {
            const cd z = ps.tsrc[i] < 0 ? cd(0, 0) : hp.table[ps.tsrc[i]];
            T->tab[i] = make_double2(z.real(), z.imag());
        }
        std::copy(ps.subs.begin(), ps.subs.end(), T->s);
        ntab = std::max(ntab, T->ntab);
        qs.progs.push_back(std::move(T));
    }
    qs.smem = smem_of(k, ntab);
    // threads: the items in as few rounds of at most 256 as they need, a multiple of 32
    const int items = int(pw[k]) / kQ3States, rounds = (items + kQ3Threads - 1) / kQ3Threads;
    qs.threads = ((items + rounds - 1) / rounds + 31) / 32 * 32;
    // the block sums use the tile buffers
    if (size_t(qs.threads) * kMaxK > size_t(2) * size_t(pw[k])) { qs.progs.clear(); return false; }
    return true;
}

}   // namespace pned
