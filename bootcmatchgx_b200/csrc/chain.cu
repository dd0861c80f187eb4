// chain.cu -- chains of l1-Jacobi sweeps of a small level in one thread-block cluster (sm_100a).
//
// A coarse level's sweep takes less time than its launch: the coarsest level runs 20 of them in a
// row per cycle (relaxnumber_coarse), 3.3 us each as dependent launches, whatever the level's size.
// Here one cluster of up to 16 blocks runs the whole chain. Every block owns R consecutive rows and
// keeps their entries on chip for all sweeps, in slices of one warp with the columns
// renumbered: the block's own rows, then the other blocks' rows that its rows use (its halo), then
// a slot that stays zero for the padding. After each sweep a block stores the new values that other
// blocks' halos hold into their shared memory (only those, from a list made at set-up) and the
// hardware cluster barrier orders them before the next sweep. The row's lanes (S, the level's threads
// per row), the order of their additions and the update are k_rowop<S>'s, so the iterates are its
// own bit for bit.
// The entries stay in registers for the chain; a sweep is then bound by the bank conflicts of the
// gathers from shared memory (about 7 cycles a warp and entry) and by the exchange and barrier (0.35 us
// of barrier). 20 sweeps of 1,950 rows of 7 entries take 17 us instead of 69 as dependent launches, of
// 3,300 irregular rows 31 instead of 73 (42 with the entries read from shared memory by 1,024 threads;
// 60 with 8 blocks instead of 16), of 7,900 rows 57. The rest is the launch and the entries' load, about
// 8 us, which is why a short chain must be small to gain (chain_pays).
#include "internal.h"
#include "rowops.cuh"

#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace bcmgx {

constexpr int kChThreads = 512;
constexpr int kChWarps = kChThreads / 32;
constexpr int kChHeld = 32;              // entries a lane holds in registers at most, over its slices
constexpr int kChSlices = 4;             // slices a warp at most
constexpr int kChPush = 3;               // push entries a thread held in registers
constexpr int kChCtas = 16;              // blocks of the largest cluster (beyond 8: not portable, asked for below)
constexpr int kChSmem = 226 * 1024;      // dynamic shared memory of a block at most
constexpr int kChMaxRows = 2047;         // rows of a block at most (11 bits of a push entry)
constexpr int kChHalo = 8192;            // halo slots and push entries of a block at most

// Per block: sizes, and its arrays at rank * (cap) of the plan's buffers.
struct alignas(16) ChainSizes {
    int entries, halo, push, slices;
    int width;   // steps of the widest slice
};
// and after them (while the plan is made): every block's halo slots by the block that owns their rows
struct ChainNeeds {
    int of[kChCtas];
};

template <typename T>
struct ChainArgs {
    int n, R, ecap, pcap, scap;
    const ChainSizes* sizes;
    const T* val;                  // entries of the slices: lane l of step k of slice s at sptr[s] + 32 k + l
    const unsigned short* idx;     // their local columns
    const unsigned* push;          // own row | block << 11 | halo slot << 15
    const int* sptr;               // first entry of every slice
    int off_f, off_M, off_x1, off_val, off_idx;   // shared-memory layout (bytes; -1: not there); x0 at 0
};

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// the address of the same shared-memory location in block `cta` of the cluster
__device__ __forceinline__ unsigned map_cta(unsigned addr, unsigned cta)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void st_cluster(unsigned a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void ch_copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

extern __shared__ __align__(128) unsigned char ch_smem[];

// k >= 2 sweeps of the level from src (from a zero iterate when src is null) into dst. One cluster. A
// warp owns up to NS slices (slices wid, wid + kChWarps, ...) and holds their first ST entries a
// lane in registers for the whole chain; longer rows read the rest from shared memory, where the
// entries are only when some row is that long (off_val >= 0).
template <int S, typename T, int NS, int ST>
__global__ void __launch_bounds__(kChThreads, 1) k_chain_cluster(ChainArgs<T> a, const T* __restrict__ f,
    const T* __restrict__ M, const T* __restrict__ src, T* __restrict__ dst, int k, const int* __restrict__ skip)
{
    using WT = typename Wider<T>::type;
    const unsigned rank = cluster_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const ChainSizes z = a.sizes[rank];
    const int r0 = (int)rank * a.R, nr = max(0, min(a.R, a.n - r0));
    T* const x0 = (T*)ch_smem;
    T* const x1 = (T*)(ch_smem + a.off_x1);
    T* fs = (T*)(ch_smem + a.off_f);
    T* Ms = (T*)(ch_smem + a.off_M);
    const int zero = a.R + z.halo;   // the slot that stays zero
    // the plan and the divisors are written during set-up only: they are read before the wait
    const T* gv = a.val + (size_t)rank * a.ecap;
    const unsigned short* gi = a.idx + (size_t)rank * a.ecap;
    if (a.off_val >= 0) {
        for (int i = tid; i < z.entries * (int)sizeof(T) / 16; i += kChThreads) ch_copy16(ch_smem + a.off_val + 16 * i, (const unsigned char*)gv + 16 * i);
        for (int i = tid; i < z.entries / 8; i += kChThreads) ch_copy16(ch_smem + a.off_idx + 16 * i, (const unsigned char*)gi + 16 * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    T v[NS][ST];
    unsigned ix[NS][ST / 2];   // two local columns a word
    int b[NS], e[NS];
#pragma unroll
    for (int t = 0; t < NS; t++) {
        const int sl = wid + t * kChWarps;
        b[t] = e[t] = 0;
        if (sl < z.slices) {
            b[t] = __ldg(a.sptr + (size_t)rank * a.scap + sl);
            e[t] = __ldg(a.sptr + (size_t)rank * a.scap + sl + 1);
        }
#pragma unroll
        for (int q = 0; q < ST; q++) {
            const int j = b[t] + 32 * q + lane;
            const bool in = j < e[t];
            v[t][q] = in ? __ldg(gv + j) : T(0);
            const unsigned c = in ? __ldg(gi + j) : (unsigned)zero;
            if (q & 1) ix[t][q / 2] |= c << 16;
            else ix[t][q / 2] = c;
        }
    }
    // the values that other blocks hold: kChPush of a thread's in registers, as the own row and the
    // address in the other block's first buffer
    int prow[kChPush];
    unsigned padr[kChPush];
    const unsigned* gp = a.push + (size_t)rank * a.pcap;
    const unsigned xa = (unsigned)__cvta_generic_to_shared(x0) + (unsigned)(a.R * (int)sizeof(T));
    auto push_addr = [&](unsigned w) { return map_cta(xa + (w >> 15) * (unsigned)sizeof(T), (w >> 11) & 15u); };
#pragma unroll
    for (int q = 0; q < kChPush; q++) {
        const int j = tid + q * kChThreads;
        prow[q] = -1;
        padr[q] = 0u;
        if (j < z.push) {
            const unsigned w = __ldg(gp + j);
            prow[q] = (int)(w & 2047u);
            padr[q] = push_addr(w);
        }
    }
    for (int i = tid; i < nr; i += kChThreads) Ms[i] = __ldg(M + r0 + i);
    if (tid == 0) x0[zero] = x1[zero] = T(0);
    cluster_arrive();   // every block has started before any stores into another's shared memory
    dep_wait();
    dep_release();
    const bool stop = skip && *skip;   // the same for every block: no kernel writes it meanwhile
    if (!stop) {
        for (int i = tid; i < nr; i += kChThreads) {
            const T fi = f[r0 + i];
            fs[i] = fi;
            x0[i] = src ? src[r0 + i] : (T)((WT)fi / (WT)Ms[i]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    cluster_wait();
    if (stop) return;
    const int sweeps = src ? k : k - 1;
    const T* vs = (const T*)(ch_smem + max(a.off_val, 0));
    const unsigned short* is = (const unsigned short*)(ch_smem + max(a.off_idx, 0));
    const int sub = lane / S;
    for (int it = 0; it < sweeps; it++) {
        T* const xc = (it & 1) ? x1 : x0;
        T* const xn = (it & 1) ? x0 : x1;
        const unsigned shift = (it & 1) ? (unsigned)a.off_x1 : 0u;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kChPush; q++)
            if (prow[q] >= 0) st_cluster(padr[q] + shift, xc[prow[q]]);
        for (int j = tid + kChPush * kChThreads; j < z.push; j += kChThreads) {
            const unsigned w = __ldg(gp + j);
            st_cluster(push_addr(w) + shift, xc[w & 2047u]);
        }
        cluster_arrive();
        cluster_wait();
        const bool last = it == sweeps - 1;
#pragma unroll
        for (int t = 0; t < NS; t++) {
            if (b[t] == e[t]) continue;   // the warp's slices end here (a slice holds its rows' diagonals)
            const int row = (wid + t * kChWarps) * (32 / S) + sub;
            T x[ST];
#pragma unroll
            for (int q = 0; q < ST; q++) x[q] = xc[(q & 1) ? ix[t][q / 2] >> 16 : ix[t][q / 2] & 0xffffu];
            T s = 0;
#pragma unroll
            for (int q = 0; q < ST; q++) s += v[t][q] * x[q];
            for (int j = b[t] + 32 * ST + lane; j < e[t]; j += 32) s += vs[j] * xc[is[j]];
            s = subwarp_sum<S>(s);
            if ((lane & (S - 1)) == 0 && row < nr) {
                const T o = (T)(((-s + fs[row]) / Ms[row]) + xc[row]);
                if (last) dst[r0 + row] = o;
                else xn[row] = o;
            }
        }
    }
}

// The halo columns of block `rank` in shared memory, by all its threads: the bits of the other blocks'
// columns that its rows use (ascending: the halo's slots), their count before each word; returns it whole.
struct ChainHalo {
    unsigned bits[(kChCtas * (kChMaxRows + 1)) / 32];
    int base[(kChCtas * (kChMaxRows + 1)) / 32 + 1];
    __device__ __forceinline__ int build(int n, int R, int rank, const int* __restrict__ row, const int* __restrict__ col)
    {
        const int tid = threadIdx.x, words = (n + 31) / 32, r0 = rank * R, r1 = min(r0 + R, n);
        for (int i = tid; i < words; i += kChThreads) bits[i] = 0u;
        __syncthreads();
        for (int r = r0 + tid; r < r1; r += kChThreads)
            for (int j = row[r]; j < row[r + 1]; j++) {
                const int c = col[j];
                if (c < r0 || c >= r0 + R) atomicOr(&bits[c >> 5], 1u << (c & 31));
            }
        __syncthreads();
        if (tid < 32) {   // one warp scans the words' counts
            int run = 0;
            for (int w0 = 0; w0 < words; w0 += 32) {
                const int w = w0 + tid, c = w < words ? __popc(bits[w]) : 0;
                int x = c;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (tid >= o) x += y;
                }
                if (w < words) base[w] = run + x - c;
                run += __shfl_sync(0xffffffffu, x, 31);
            }
            if (tid == 0) base[words] = run;
        }
        __syncthreads();
        return base[words];
    }
    // halo columns below c: the slot of a column that is one
    __device__ __forceinline__ int slot(int c) const { return base[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u)); }
    __device__ __forceinline__ int slots_below(int c, int n, int H) const { return c < n ? slot(c) : H; }
};

// The plan's sizes, a block of the grid for each of the cluster's: its slices' widths (sptr) and its halo.
// Neither this nor k_chain_fill is a cluster: where none of the wanted size can run, set-up goes on without.
__global__ void __launch_bounds__(kChThreads) k_chain_sizes(int n, int R, int S, int scap, const int* __restrict__ row,
    const int* __restrict__ col, int* __restrict__ sptr, ChainSizes* sizes, ChainNeeds* needs)
{
    __shared__ ChainHalo halo;
    const int rank = blockIdx.x, tid = threadIdx.x;
    const int r0 = rank * R, nr = max(0, min(R, n - r0)), rs = 32 / S, slices = (nr + rs - 1) / rs;
    const int H = halo.build(n, R, rank, row, col);
    if (tid < (int)gridDim.x) needs[rank].of[tid] = halo.slots_below((tid + 1) * R, n, H) - halo.slots_below(tid * R, n, H);
    if (tid < 32) {
        int at = 0, widest = 0;
        for (int t0 = 0; t0 < slices; t0 += 32) {
            const int t = t0 + tid;
            int w = 0;
            if (t < slices)
                for (int i = 0; i < rs; i++) {
                    const int r = t * rs + i;
                    if (r < nr) w = max(w, (row[r0 + r + 1] - row[r0 + r] + S - 1) / S);
                }
            widest = max(widest, w);
            int x = 32 * w;
            const int c = x;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (tid >= o) x += y;
            }
            if (t < slices) sptr[(size_t)rank * scap + t] = at + x - c;
            at += __shfl_sync(0xffffffffu, x, 31);
        }
        widest = __reduce_max_sync(0xffffffffu, widest);
        if (tid == 0) {
            sptr[(size_t)rank * scap + slices] = at;
            sizes[rank].entries = at;
            sizes[rank].halo = H;
            sizes[rank].slices = slices;
            sizes[rank].width = widest;
        }
    }
}

// The plan's entries and push lists, once the sizes are known to fit ecap and pcap a block.
template <typename T>
__global__ void __launch_bounds__(kChThreads) k_chain_fill(int n, int R, int S, int ecap, int pcap, int scap,
    const int* __restrict__ row, const int* __restrict__ col, const T* __restrict__ val, const int* __restrict__ sptr,
    T* __restrict__ pval, unsigned short* __restrict__ pidx, unsigned* __restrict__ push, ChainSizes* sizes, const ChainNeeds* __restrict__ needs)
{
    __shared__ ChainHalo halo;
    __shared__ int at[kChCtas];
    const int rank = blockIdx.x, tid = threadIdx.x;
    const int r0 = rank * R, nr = max(0, min(R, n - r0)), rs = 32 / S, slices = (nr + rs - 1) / rs;
    const int H = halo.build(n, R, rank, row, col);
    // An owner's list goes by the block that needs the value and by its slot there, so that consecutive
    // threads store to consecutive addresses of one block (scattered, an FP64 solve of 127x93x75 rows took 2.4 %
    // longer). at[own]: where the owner's list has this block's slots, less the first of them.
    if (tid < (int)gridDim.x) {
        int o = 0, all = 0;
        for (int c = 0; c < (int)gridDim.x; c++) {
            if (c == rank) o = all;
            all += needs[c].of[tid];
        }
        at[tid] = o - halo.slots_below(tid * R, n, H);
        if (tid == rank) sizes[rank].push = all;
    }
    __syncthreads();
    for (int w = tid; w < (n + 31) / 32; w += kChThreads) {
        unsigned m = halo.bits[w];
        for (int slot = halo.base[w]; m; slot++, m &= m - 1u) {
            const int c = 32 * w + __ffs((int)m) - 1, own = c / R;
            push[(size_t)own * pcap + at[own] + slot] = (unsigned)(c - own * R) | ((unsigned)rank << 11) | ((unsigned)slot << 15);
        }
    }
    for (int t = tid >> 5; t < slices; t += kChThreads / 32) {
        const int lane = tid & 31, r = t * rs + lane / S;
        const int b = r < nr ? row[r0 + r] : 0, e = r < nr ? row[r0 + r + 1] : 0;
        const int o = sptr[(size_t)rank * scap + t], kk = (sptr[(size_t)rank * scap + t + 1] - o) / 32;
        for (int q = 0; q < kk; q++) {
            const int j = b + q * S + (lane & (S - 1));
            int ix = R + H;
            T v = T(0);
            if (j < e) {
                const int c = col[j];
                v = val[j];
                ix = c >= r0 && c < r0 + R ? c - r0 : R + halo.slot(c);
            }
            pval[(size_t)rank * ecap + o + 32 * q + lane] = v;
            pidx[(size_t)rank * ecap + o + 32 * q + lane] = (unsigned short)ix;
        }
    }
}

// Whether a chain of k sweeps is one launch: from 8 sweeps up on every level that fits (chain_fits); the
// usual 4 only on levels of at most 50,000 entries (at 105,000 entries 12.9 us against 13.6, and 16 SMs
// against the whole GPU beyond).
static bool chain_pays(const DevCsr& A, int k) { return k >= 8 || (k >= 2 && A.nnz <= 50000); }

// Whether a block's warps have few enough slices of the level: two at most, or four on a level of at most 82,000
// entries. A third and fourth cost a sweep more than its launch does. One cycle whose coarsest level takes 20
// sweeps (8), launches -> cluster: 8,000 rows of 24 entries 109 -> 98 us (78 -> 74), 7,641 irregular rows 99 -> 96
// (69 -> 67); above two slices 8,870 irregular rows would go 99 -> 105 (70 -> 71), 9,261 of 24 entries 109 -> 124
// (79 -> 85) and 13,824 of 7 99 -> 101 (70 -> 72), but 12,167 of 7 (81,995 entries) 98 -> 96 (70 -> 69).
static bool chain_fits(const DevCsr& A, int R, int S)
{
    const int slices = ceil_div(R, 32 / S);
    return slices <= 2 * kChWarps || (slices <= kChSlices * kChWarps && A.nnz <= 82000);
}

template <typename K>
static cudaLaunchConfig_t cluster_config(K kern, int ctas, size_t smem, cudaStream_t s, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kChThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    BCMGX_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    ensure_smem_limit((const void*)kern, smem);
    return cfg;
}

// Runs F(kernel) with the chain kernel for S threads per row, ns slices a warp and st entries of each
// in registers (the least compiled forms that have room; ns * st <= kChHeld).
template <typename T, typename F>
static void with_chain_kernel(int S, int ns, int st, F&& go)
{
    auto form = [&](auto s_) {
        constexpr int SS = decltype(s_)::value;
        if (ns <= 1 && st > 16) go(k_chain_cluster<SS, T, 1, 32>);
        else if (ns <= 1 && st > 8) go(k_chain_cluster<SS, T, 1, 16>);
        else if (ns <= 1) go(k_chain_cluster<SS, T, 1, 8>);
        else if (ns <= 2 && st > 8) go(k_chain_cluster<SS, T, 2, 16>);
        else if (ns <= 2) go(k_chain_cluster<SS, T, 2, 8>);
        else go(k_chain_cluster<SS, T, kChSlices, 8>);
    };
    switch (S) {
    case 1: form(std::integral_constant<int, 1>()); break;
    case 2: form(std::integral_constant<int, 2>()); break;
    case 4: form(std::integral_constant<int, 4>()); break;
    case 8: form(std::integral_constant<int, 8>()); break;
    default: form(std::integral_constant<int, 16>()); break;
    }
}

template <typename T>
static bool build_chain_t(Level& V, const T* val, bool fill, cudaStream_t s)
{
    const DevCsr& A = V.A;
    const int n = A.n, S = A.tpr;
    std::unique_ptr<ChainPlan> P(new ChainPlan());
    // blocks: one while its warps have a slice each at most, else as many as leave 4 slices a block,
    // up to the largest cluster (fewer rows a block cost less than the larger barrier)
    const long slices = ((long)n * S + 31) / 32;
    int ctas = 1;
    if (slices > kChWarps)
        while (ctas < kChCtas && slices > 4L * ctas) ctas *= 2;
    P->ctas = ctas;
    P->n = n;
    P->R = ((n + ctas - 1) / ctas + 1) / 2 * 2;
    P->S = S;
    P->f32 = sizeof(T) == 4;
    if (P->R > kChMaxRows) return false;
    if (!chain_fits(A, P->R, S)) return false;
    P->scap = (P->R * S / 32 + 2 + 3) / 4 * 4 + 4;
    P->sptr.alloc((size_t)ctas * P->scap, s);
    const size_t sizes_bytes = (size_t)ctas * sizeof(ChainSizes);
    P->sizes.alloc((sizes_bytes + (size_t)ctas * sizeof(ChainNeeds)) / sizeof(int), s);
    ChainSizes* const sizes = (ChainSizes*)P->sizes.p;
    ChainNeeds* const needs = (ChainNeeds*)(sizes + ctas);
    note_launch();
    k_chain_sizes<<<ctas, kChThreads, 0, s>>>(n, P->R, S, P->scap, A.row.p, A.col.p, P->sptr.p, sizes, needs);
    BCMGX_CHECK_LAUNCH();
    std::vector<unsigned char> host(sizes_bytes + (size_t)ctas * sizeof(ChainNeeds));
    BCMGX_CUDA(cudaMemcpyAsync(host.data(), sizes, host.size(), cudaMemcpyDeviceToHost, s));
    BCMGX_CUDA(cudaStreamSynchronize(s));
    const ChainSizes* z = (const ChainSizes*)host.data();
    const ChainNeeds* zn = (const ChainNeeds*)(z + ctas);
    int E = 0, H = 0, N = 0, W = 0;
    for (int c = 0; c < ctas; c++) {
        int push = 0;
        for (int b = 0; b < ctas; b++) push += zn[b].of[c];
        if (z[c].entries > kChSmem / (int)(sizeof(T) + 2) || z[c].halo > kChHalo || push > kChHalo) return false;
        P->pcap = std::max(P->pcap, push);
        E = std::max(E, z[c].entries);
        H = std::max(H, z[c].halo);
        N = std::max(N, z[c].slices);
        W = std::max(W, z[c].width);
    }
    P->ns = (N + kChWarps - 1) / kChWarps;
    // shared memory: both iterates (own rows, halo, the zero slot), f, M, and the entries of levels
    // with rows longer than the registers hold
    auto up16 = [](size_t b) { return (b + 15) / 16 * 16; };
    size_t o = up16((size_t)(P->R + H + 1) * sizeof(T));
    P->off_x1 = (int)o;
    o += up16((size_t)(P->R + H + 1) * sizeof(T));
    P->off_f = (int)o;
    o += up16((size_t)P->R * sizeof(T));
    P->off_M = (int)o;
    o += up16((size_t)P->R * sizeof(T));
    P->st = std::min(W, kChHeld / (P->ns <= 1 ? 1 : P->ns <= 2 ? 2 : kChSlices));
    if (W > P->st) {
        P->off_val = (int)o;
        o += up16((size_t)E * sizeof(T));
        P->off_idx = (int)o;
        o += up16((size_t)E * 2);
    }
    P->smem = o;
    if (o > (size_t)kChSmem) return false;
    int fit = 0;
    with_chain_kernel<T>(S, P->ns, P->st, [&](auto kern) {
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t cfg = cluster_config(kern, ctas, o, s, at);
        if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            fit = 0;
        }
    });
    if (fit < 1) return false;
    if (!fill) return true;
    P->ecap = E;   // whole slices: every block's entries start on a 16-byte boundary
    P->val.alloc((size_t)ctas * E * sizeof(T), s);
    P->idx.alloc((size_t)ctas * E, s);
    P->push.alloc((size_t)ctas * P->pcap, s);
    note_launch();
    k_chain_fill<T><<<ctas, kChThreads, 0, s>>>(n, P->R, S, P->ecap, P->pcap, P->scap, A.row.p, A.col.p, val, P->sptr.p,
        (T*)P->val.p, P->idx.p, P->push.p, sizes, needs);
    BCMGX_CHECK_LAUNCH();
    V.chain = std::move(P);
    return true;
}

bool chain_wanted(const DevCsr& A, bool f32, int k)
{
    const char* env = std::getenv("BCMGX_CHAIN");
    if ((env && env[0] == '0') || !chain_pays(A, k)) return false;
    if (A.stencil || A.sliced || A.staged) return false;   // levels tuned to stream over the whole GPU
    if (A.n <= 0 || A.m != A.n || A.n > kChCtas * kChMaxRows || A.tpr > 16) return false;
    return A.nnz * (int64_t)((f32 ? 4 : 8) + 2) <= (int64_t)kChCtas * kChSmem;
}

bool build_chain(Level& V, bool f32, bool fill, cudaStream_t s)
{
    const DevCsr& A = V.A;
    if (f32) return A.val32.p && build_chain_t<float>(V, A.val32.p, fill, s);
    return build_chain_t<double>(V, A.val.p, fill, s);
}

template <typename T>
static void run_chain_t(const Level& V, const T* M, int k, const T* f, const T* src, T* dst, const int* skip, cudaStream_t s)
{
    const ChainPlan& P = *V.chain;
    ChainArgs<T> a {};
    a.n = P.n;
    a.R = P.R;
    a.ecap = P.ecap;
    a.pcap = P.pcap;
    a.scap = P.scap;
    a.sizes = (const ChainSizes*)P.sizes.p;
    a.val = (const T*)P.val.p;
    a.idx = P.idx.p;
    a.push = P.push.p;
    a.sptr = P.sptr.p;
    a.off_f = P.off_f;
    a.off_M = P.off_M;
    a.off_x1 = P.off_x1;
    a.off_val = P.off_val;
    a.off_idx = P.off_idx;
    with_chain_kernel<T>(P.S, P.ns, P.st, [&](auto kern) {
        cudaLaunchAttribute at[2];
        cudaLaunchConfig_t cfg = cluster_config(kern, P.ctas, P.smem, s, at);
        if (dep_launch_enabled(0)) {
            at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.numAttrs = 2;
        }
        note_launch();
        BCMGX_CUDA(cudaLaunchKernelEx(&cfg, kern, a, f, M, src, dst, k, skip));
    });
}

bool run_chain(const Level& V, bool f32, int k, const void* f, const void* src, void* dst, const int* skip, cudaStream_t s)
{
    if (!V.chain || V.chain->f32 != f32 || !chain_pays(V.A, k)) return false;
    if (f32) run_chain_t<float>(V, V.M32.p, k, (const float*)f, (const float*)src, (float*)dst, skip, s);
    else run_chain_t<double>(V, V.M.p, k, (const double*)f, (const double*)src, (double*)dst, skip, s);
    return true;
}

}  // namespace bcmgx
