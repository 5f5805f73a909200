// fgpe_group.cuh -- grouped passes: one launch advances every instance of a
// batch that shares a grid shape (q2D, both axes of a size the size-
// specialised kernels cover), instead of one launch per instance.
//
// A group's instances differ in their physics (TAU, GAMMA, ALPHA, DT) and
// state buffers, described per instance by an InstDesc in device memory.  A
// launch walks the tiles of all of them: column tiles are independent
// (k_regcol_group); rows are taken in chunks of consecutive tiles (the block
// pass below) or batches (k_regrow_group) of one instance, each chunk adds
// its NORMC partial to the instance's slot for that chunk, and whoever
// completes an instance's last chunk reduces the slots in a fixed order and
// publishes the norms and next scales (as the last block of the
// single-instance row pass does), so results do not depend on timing.
#pragma once
#include "fgpe_fast.cuh"

namespace fgpe {

struct InstDesc {
    StepConst c;
    void* S;            // x-spectral state (in/out)
    void* psi;          // real-space snapshot target of mode 1
    void* prev;         // real-space snapshot target of mode 2
    double* info;       // INFO_* vector
    double* info_prev;  // receives info after a mode-2 step
    double* part;       // NORMC partials, [chunks][MS]
    unsigned* counter;  // chunks finished in the current launch (0 between)
};

struct GroupArgs {
    const InstDesc* d;
    int ninst;
    int tiles;          // tiles per instance
    int chunk;          // row pass: tiles per chunk (divides tiles)
    int snap;           // row pass: 0 none, 1 real-space state to psi, 2 to prev (+ info to info_prev)
};

// The StepConst of the tile's instance, copied into shared memory when the
// instance changes (device functions read it there rather than from global
// memory).  Callers synchronise before using it.
__device__ __forceinline__ void load_const(StepConst& dst, const StepConst& src) {
    const int nw = (int)(sizeof(StepConst) / 4);
    const unsigned* s = (const unsigned*)&src;
    unsigned* d = (unsigned*)&dst;
    for (int i = threadIdx.x; i < nw; i += blockDim.x) d[i] = s[i];
}

// Completion of one instance's NORMC after a chunk has written its slot.
template <int MS>
__device__ void finish_group_norms(const InstDesc& D, const StepConst& c, int nchunk, bool keep_prev,
                                   double* red) {
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = (atomicAdd(D.counter, 1u) == (unsigned)nchunk - 1u);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double acc[MS];
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    for (int b = threadIdx.x; b < nchunk; b += blockDim.x) {
#pragma unroll
        for (int m = 0; m < MS; ++m) acc[m] += __ldcg(D.part + (size_t)b * MS + m);
    }
    block_sum<MS>(acc, red, red + 32 * MS);
    if (threadIdx.x == 0) {
        double tot = 0, n[MS], sc[MS];
        double* info = D.info;
        for (int m = 0; m < MS; ++m) { n[m] = red[32 * MS + m]; tot += n[m]; info[INFO_NORM + m] = n[m]; }
        info[INFO_TOTAL] = tot;
        sink_norms<MS>(c, n);
        const int rc = compute_scales<MS>(c, n, info + INFO_SIG, sc);
        bool bad = !(tot == tot) || !(tot < 1e300);
        for (int m = 0; m < MS; ++m) { info[INFO_SC + m] = sc[m]; bad = bad || !(sc[m] == sc[m]); }
        if (bad) info[INFO_ERR] = 1.0;
        if (rc) info[INFO_ERR] = (double)rc;
        if (keep_prev)
            for (int i = 0; i < INFO_LEN; ++i) D.info_prev[i] = info[i];
        *D.counter = 0u;
    }
    __syncthreads();
}

// The same by one warp, whose NORMC terms (one value per lane and component)
// are those of the instance's chunk `slot`; acc starts again from zero.
template <int MS>
__device__ __forceinline__ void warp_finish_norms(const InstDesc& D, int slot, int nslots, bool keep_prev, double (&acc)[MS]) {
    const int lane = threadIdx.x & 31;
    auto warp_sum = [&](double (&v)[MS]) {
#pragma unroll
        for (int m = 0; m < MS; ++m)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[m] += __shfl_xor_sync(0xffffffffu, v[m], o);
    };
    warp_sum(acc);
    int last = 0;
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MS; ++m) D.part[(size_t)slot * MS + m] = acc[m];
        __threadfence();
        last = atomicAdd(D.counter, 1u) == (unsigned)nslots - 1u;
    }
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
    for (int b = lane; b < nslots; b += 32) {
#pragma unroll
        for (int m = 0; m < MS; ++m) acc[m] += __ldcg(D.part + (size_t)b * MS + m);
    }
    warp_sum(acc);
    if (lane == 0) {
        double tot = 0, n[MS], sc[MS];
        double* info = D.info;
        for (int m = 0; m < MS; ++m) { n[m] = acc[m]; tot += n[m]; info[INFO_NORM + m] = n[m]; }
        info[INFO_TOTAL] = tot;
        sink_norms<MS>(D.c, n);
        const int rc = compute_scales<MS>(D.c, n, info + INFO_SIG, sc);
        bool bad = !(tot == tot) || !(tot < 1e300);
        for (int m = 0; m < MS; ++m) { info[INFO_SC + m] = sc[m]; bad = bad || !(sc[m] == sc[m]); }
        if (bad) info[INFO_ERR] = 1.0;
        if (rc) info[INFO_ERR] = (double)rc;
        if (keep_prev)
            for (int i = 0; i < INFO_LEN; ++i) D.info_prev[i] = info[i];
        *D.counter = 0u;
    }
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    __syncwarp();
}

// ------------------------------------------------------------ row pass
// ROW_FULL of every instance: tiles of R x-lines, chunks of g.chunk tiles.
template <typename T, int MS, int N, int R, int TH, int NBUF = FGPE_ROW_NBUF>
__global__ void __launch_bounds__(TH, row_minb(TH)) k_row_group(GroupArgs g) {
    using RT = RowTile<N, MS * R>;
    constexpr int LP = RT::LP;
    constexpr int TILE = MS * R * LP;
    constexpr int NCH = MS * R * N;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* bufs = (cx<T>*)smraw;
    __shared__ double red[32 * (MS + 1)];
    __shared__ double bsum[MS];
    __shared__ StepConst c;
    const int nci = g.tiles / g.chunk;            // chunks per instance
    const int nchunks = g.ninst * nci;
    // k-th tile of this block: chunk blockIdx.x + (k / chunk) * gridDim.x
    auto tile_of = [&](int k, int& inst, int& lt) -> bool {
        const int q = k / g.chunk;
        const int chunk = blockIdx.x + q * gridDim.x;
        if (chunk >= nchunks) return false;
        inst = chunk / nci;
        lt = (chunk - inst * nci) * g.chunk + (k - q * g.chunk);
        return true;
    };
    auto issue = [&](int inst, int lt, cx<T>* dst) {
        const InstDesc& D = g.d[inst];
        const cx<T>* src = (const cx<T>*)D.S;
        const long long np = D.c.npts;
        const int row0 = lt * R;
        for (int ch = threadIdx.x; ch < NCH; ch += TH) {
            const int x = ch % N;
            const int q = ch / N;
            const int r = q % R, m = q / R;
            cp_elem<T>(dst + (m * R + r) * LP + x + (x >> 3), src + (size_t)m * np + (size_t)(row0 + r) * N + x);
        }
    };
    double acc[MS];
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    int inst = 0, lt = 0, cur_inst = -1;
    bool have = tile_of(0, inst, lt);
    if (NBUF == 2) {
        if (have) issue(inst, lt, bufs);
        cp_commit();
    }
    for (int k = 0; have; ++k) {
        cx<T>* cur = bufs + (NBUF == 2 ? (k & 1) * TILE : 0);
        int ninst = 0, nlt = 0;
        const bool nxt = tile_of(k + 1, ninst, nlt);
        if (inst != cur_inst) {
            __syncthreads();                       // nobody still reads the old constants
            load_const(c, g.d[inst].c);
            cur_inst = inst;
        }
        if (NBUF == 2) {
            if (nxt) issue(ninst, nlt, bufs + ((k + 1) & 1) * TILE);
            cp_commit();
            cp_wait<1>();
        } else {
            issue(inst, lt, cur);
            cp_commit();
            cp_wait<0>();
        }
        __syncthreads();
        const InstDesc& D = g.d[inst];
        const long long np = c.npts;
        const cx<T>* twx = (const cx<T>*)c.twx;
        const int row0 = lt * R;
        cx<T>* snap = g.snap == 1 ? (cx<T>*)D.psi : g.snap == 2 ? (cx<T>*)D.prev : nullptr;
        ct_fft<T, true, N, MS * R, TH, RT>(cur, twx);
        for (int p = threadIdx.x; p < R * N; p += TH) {
            const int x = p % N, r = p / N;
            const int row = row0 + r;
            const int j = row % c.ny, kk = row / c.ny;
            cx<T> v[MS];
#pragma unroll
            for (int m = 0; m < MS; ++m) v[m] = cur[(m * R + r) * LP + x + (x >> 3)];
            const cx<T> eV = pot_phase<T>(c, x, j, kk);
            apply_se<T, MS>(c, v);
            apply_sp<T, MS>(c, eV, v);
            double w = c.wx[x] * c.wy[j];
#pragma unroll
            for (int m = 0; m < MS; ++m) {
                acc[m] += w * ((double)v[m].x * (double)v[m].x + (double)v[m].y * (double)v[m].y);
                cur[(m * R + r) * LP + x + (x >> 3)] = v[m];
            }
            if (snap) {
#pragma unroll
                for (int m = 0; m < MS; ++m) snap[(size_t)m * np + (size_t)row * N + x] = v[m];
            }
        }
        __syncthreads();
        ct_fft<T, false, N, MS * R, TH, RT>(cur, twx);
        cx<T>* S = (cx<T>*)D.S;
        for (int idx = threadIdx.x; idx < MS * R * N; idx += TH) {
            const int x = idx % N, q = idx / N, r = q % R, m = q / R;
            S[(size_t)m * np + (size_t)(row0 + r) * N + x] = cur[(m * R + r) * LP + x + (x >> 3)];
        }
        __syncthreads();
        if ((k + 1) % g.chunk == 0) {
            // this block's chunk of the instance is done: publish its partial
            block_sum<MS>(acc, red, bsum);
            const int chunk = blockIdx.x + (k / g.chunk) * gridDim.x;
            if (threadIdx.x < MS) D.part[(size_t)(chunk - inst * nci) * MS + threadIdx.x] = bsum[threadIdx.x];
#pragma unroll
            for (int m = 0; m < MS; ++m) acc[m] = 0.0;
            finish_group_norms<MS>(D, c, nci, g.snap == 2, red);
        }
        inst = ninst; lt = nlt; have = nxt;
    }
    cp_wait<0>();
}

}  // namespace fgpe
