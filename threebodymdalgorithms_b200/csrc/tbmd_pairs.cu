// No-cutoff forces and energy as a matrix product: the mixed form (and its adjoint) on the tensor cores, the
// FP64 form on the FP64 matrix instruction (second part of this file).
//
// With the pair tensors T_ij = (3 r r^T - r^2) / r^5 (r = x_j - x_i, symmetric, traceless, T_ii = 0) the
// Axilrod-Teller energy of a triplet is -nu/3 tr(T_ij T_jk T_ki), so over all triplets
//   E   = -nu/18 tr(T^3)                             (T: the symmetric 3n x 3n matrix of the 3x3 blocks)
//   f_i = +dE/dx_i = nu/3 sum_j (G_ij : dT_ij/dr),   G = T T,   G_ij = sum_k T_ik T_kj
// which is the same sum over i < j < k as the pairwise sweeps (the blocks T_ii = 0 leave out repeated
// indices).  G is a dense product of 27 n^3 FLOP over i < j; the rest is O(n^2).
//
//   k_pt_panel   T for a range of k, formed in FP64 and split exactly into three bfloat16 (h + m + l holds
//                26 bits), written in the layout the matrix unit reads from shared memory
//   k_pt_gemm    tiles of G (84 x 84 particles over two SMs) by tcgen05.mma, contracted with dT/dr in the
//                same kernel
//   k_pt_reduce  each particle's force from its tiles, in a fixed order (deterministic)
//
// Bound: the tensor cores, at the power cap for large n.  n = 8192: 9.4e13 FLOP of bf16 in 70 ms, 1.35
// PFLOP/s, as much as cuBLAS sustains (AUTA's FP32 sweep took 240 ms, NATA's 541); n = 4096: 8.9 ms
// (31.5 and 79).  A pair of SMs works on one tile of 256 x 256 (cta_group::2), which halves what each loads
// of B: 48 KB a slab.  A block's 128 x 256 part is the largest whose FP32 sums fit the registers (128 a
// thread in eight warps) beside two accumulators of 256 TMEM columns, one filling while the other is added
// up (350 cycles of the 1,536 that a slab's product takes).  One block alone with the same tile of 128 x 256
// and the FP32 geometry of each row's pairs in every thread took 82 ms: 17,000 cycles of contraction an item.
//
// Accuracy.  Six products of the splits are kept (hh, hm, mh, mm, hl, lh; the rest is below 2^-26), each
// exact in FP32.  The tensor core adds into an FP32 accumulator that it truncates, so an accumulator only
// lives for 32 columns of T: the ten small products go first, the two hh steps last, and the tile is then
// added to FP32 registers with rounding.  After 512 particles at most the registers are contracted and the
// forces go on in FP64.  Relative L2 errors against FP64, product and FP32 sweep on the same inputs of 200 .. 4096
// particles: thermal lattices, forces 1.3e-7 .. 2.3e-7 (sweeps 2.0e-7 .. 2.8e-7), H d 1.5e-7 .. 2.6e-7 (3.2e-7 ..
// 4.8e-7); uniform inputs, which hang on one or two close pairs, forces 3.8e-8 .. 4.1e-7 (3.3e-8 .. 7.8e-7), H d
// 7.2e-8 .. 3.8e-7 (4.7e-8 .. 1.4e-6).  No step subtracts nearly equal numbers: a pair's force needs no difference of
// large terms even where two of the three particles nearly coincide.
//
// Three modules come from this source: 0 the mixed forces and the host's part, 1 the kernels of the mixed adjoint
// (tbmd_pairs_adjoint.cu), 2 those of the FP64 form (tbmd_pairs_fp64.cu).  The first launch of a kernel in a process loads
// its whole module, 1.24 ms for all in one, 0.44 + 0.72 and 0.36 as they are.
#ifndef TBMD_PAIRS_MODULE
#define TBMD_PAIRS_MODULE 0
#endif

#include <cuda_bf16.h>

#include <algorithm>

#include "tbmd_internal.cuh"

namespace tbmd {

// One group's kernels of module 1 (T' and the second-order terms, then G') and of module 2, and their set-up.
cudaError_t pt_init_adjoint(bool energy);
void pt_launch_adjoint(bool second, Pos pos, const PtGroup &g, const PtDev &d, bool energy, double nu, int sms, cudaStream_t st);
cudaError_t pt_init_fp64(bool energy);
void pt_launch_fp64(Pos pos, Out out, const PtPlan &plan, const PtGroup &g, const PtDev &d, double *energy, double nu,
                    int sms, cudaStream_t st);

// A row block holds 42 particles in 126 of its 128 rows, two particles side by side in six rows (x x' y y'
// z z'), so that the columns of a tile come in pairs that packed FP32 operations take at once.
constexpr int PT_PART = 42;
constexpr int PT_ROWS = 128;
constexpr int PT_SLAB_K = 32;               // matrix columns of one slab (one pipeline stage)
constexpr int PT_SPLIT_BYTES = PT_ROWS * PT_SLAB_K * 2;  // one split of a row block's slab: 8 KB
constexpr int PT_BLOCK_BYTES = 3 * PT_SPLIT_BYTES;       // all three: 24 KB, contiguous in the panel
constexpr int PT_STAGE_BYTES = 2 * PT_BLOCK_BYTES;       // one row block of A and one of B
constexpr int PT_STAGES = 3;
constexpr int PT_GEO = 2 * (PT_PART / 2) * PT_PART;      // pair geometry of a block's tile: [pair of j][i]
// 8 warps accumulate and contract, 1 loads, 1 issues the products, 2 fetch positions
constexpr int PT_WARPS = 12;
// doubles of a tile's results for row blocks of `part` particles: f_i, f_j (two blocks), energy, pad
__host__ __device__ constexpr int pt_slot(int part) { return 9 * part + 2; }
constexpr int PT_SLOT = pt_slot(PT_PART);

struct PtShared {
    unsigned char stage[PT_STAGES][PT_STAGE_BYTES];
    // (n_x n_x' n_y n_y') and (n_z n_z' r^-4 r'^-4) of particle i and two j; with the second-order terms for one
    // column block at a time, its rates behind it
    float4 geo[2][PT_GEO];
    double xj[6][2 * PT_PART], xi[6][PT_PART];  // positions of the tile's particles, and their directions
    double fi[2][PT_ROWS][3];
    float fj[8][PT_ROWS];
    double e[8];
    unsigned long long full[PT_STAGES], empty[PT_STAGES], acc_full[2], acc_empty[2], geo_full, geo_empty, drained;
    unsigned int tmem;
    int dead;
};

__device__ __forceinline__ unsigned int smem_u32(const void *p) { return (unsigned int)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long *b, unsigned int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *b, unsigned int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// Arrive on the same barrier of block `rank` of the cluster, after reads of TMEM (ordered by tcgen05.fence).
// Nothing is handed over in memory, so the arrival is relaxed: a release at cluster scope waits for the
// thread's global stores, 1,000 cycles a slab in the warps that write the tiles' results.
__device__ __forceinline__ void bar_arrive_tmem(unsigned long long *b, unsigned int rank)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, %1;\n\t"
        "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(b)),
        "r"(rank)
        : "memory");
}
// The same for a thread that has seen a bulk copy of its own block complete and passes that on: what the copy
// wrote is ordered before the arrival, for a wait with bar_try_cluster.
__device__ __forceinline__ void bar_relay_copy(unsigned long long *b, unsigned int rank)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, %1;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(b)),
        "r"(rank)
        : "memory");
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long *b, unsigned int parity)
{
    unsigned int ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// for a phase that the other block's arrivals complete: acquires what they released
__device__ __forceinline__ bool bar_try_cluster(unsigned long long *b, unsigned int parity)
{
    unsigned int ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Every wait ends: after wt.limit cycles it marks the block dead and the launch failed (*wt.err); from then on
// waits return at once, no copy or product is issued, and the loops run out.  A limit of zero gives up the first.
template <bool CLUSTER = false, class Shared>
__device__ __forceinline__ bool bar_wait(unsigned long long *b, unsigned int parity, Shared &S, const PtWait &wt)
{
    auto done = [&]() { return CLUSTER ? bar_try_cluster(b, parity) : bar_try(b, parity); };
    if (wt.limit > 0 && done()) return true;
    const long long t0 = clock64();
    if (wt.limit <= 0) {
        *(volatile int *)&S.dead = 1;
        atomicExch(wt.err, 1u);
        return false;
    }
    for (unsigned int n = 1;; ++n) {
        if (done()) return true;
        if ((n & 63u) == 0u) {
            if (*(volatile int *)&S.dead) return false;
            if (clock64() - t0 > wt.limit) {
                *(volatile int *)&S.dead = 1;
                atomicExch(wt.err, 1u);
                return false;
            }
        }
    }
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned int bytes, unsigned long long *b)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(b))
                 : "memory");
}
// Shared-memory descriptor of an operand stored without swizzle, K contiguous in 16-byte chunks: the next
// chunk of 8 columns is 128 bytes on, the next group of 8 rows 512.
__device__ __forceinline__ unsigned long long operand_desc(unsigned int addr)
{
    return (unsigned long long)((addr >> 4) & 0x3fffu) | (unsigned long long)(128 >> 4) << 16 |
           (unsigned long long)(512 >> 4) << 32 | 1ull << 46;
}
// D FP32, A and B bfloat16, both K-major, 256 x 256 over the two blocks of a cluster: each holds 128 rows of
// A, 128 of B, and 128 rows x 256 columns of D in its TMEM
constexpr unsigned int PT_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
__device__ __forceinline__ void mma_bf16(unsigned int d, unsigned long long a, unsigned long long b, unsigned int acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(PT_IDESC), "r"(acc)
        : "memory");
}
// the barrier at this address in both blocks gets an arrival when the products issued so far are done
__device__ __forceinline__ void mma_commit(unsigned long long *b)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(b)),
                 "h"((unsigned short)3)
                 : "memory");
}
// the same for this block's barrier alone
__device__ __forceinline__ void mma_commit_local(unsigned long long *b)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b)) : "memory");
}
// 64 columns of this warp's 32 TMEM lanes
#define TM_LD64(v, addr)                                                                                       \
    asm volatile(                                                                                              \
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%1" \
        "7,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%4" \
        "2,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"       \
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),                              \
          "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),                            \
          "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]),                        \
          "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),                        \
          "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]),                        \
          "=f"(v[30]), "=f"(v[31]), "=f"(v[32]), "=f"(v[33]), "=f"(v[34]), "=f"(v[35]),                        \
          "=f"(v[36]), "=f"(v[37]), "=f"(v[38]), "=f"(v[39]), "=f"(v[40]), "=f"(v[41]),                        \
          "=f"(v[42]), "=f"(v[43]), "=f"(v[44]), "=f"(v[45]), "=f"(v[46]), "=f"(v[47]),                        \
          "=f"(v[48]), "=f"(v[49]), "=f"(v[50]), "=f"(v[51]), "=f"(v[52]), "=f"(v[53]),                        \
          "=f"(v[54]), "=f"(v[55]), "=f"(v[56]), "=f"(v[57]), "=f"(v[58]), "=f"(v[59]),                        \
          "=f"(v[60]), "=f"(v[61]), "=f"(v[62]), "=f"(v[63])                                                   \
        : "r"(addr))
// the loaded registers hold their values from here on
#define TM_WAIT64(v)                                                                             \
    asm volatile("tcgen05.wait::ld.sync.aligned;"                                                \
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),       \
                   "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]),     \
                   "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15]), "+f"(v[16]), "+f"(v[17]), \
                   "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]), "+f"(v[22]), "+f"(v[23]), \
                   "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27])                            \
                 :                                                                               \
                 : "memory");                                                                    \
    asm volatile(""                                                                              \
                 : "+f"(v[28]), "+f"(v[29]), "+f"(v[30]), "+f"(v[31]), "+f"(v[32]), "+f"(v[33]), \
                   "+f"(v[34]), "+f"(v[35]), "+f"(v[36]), "+f"(v[37]), "+f"(v[38]), "+f"(v[39]), \
                   "+f"(v[40]), "+f"(v[41]), "+f"(v[42]), "+f"(v[43]), "+f"(v[44]), "+f"(v[45]), \
                   "+f"(v[46]), "+f"(v[47]), "+f"(v[48]), "+f"(v[49]), "+f"(v[50]), "+f"(v[51]), \
                   "+f"(v[52]), "+f"(v[53]), "+f"(v[54]), "+f"(v[55])                            \
                 :                                                                               \
                 : "memory");                                                                    \
    asm volatile(""                                                                              \
                 : "+f"(v[56]), "+f"(v[57]), "+f"(v[58]), "+f"(v[59]), "+f"(v[60]), "+f"(v[61]), \
                   "+f"(v[62]), "+f"(v[63])                                                      \
                 :                                                                               \
                 : "memory")

// two FP32 values in one register pair, and the packed operations on them
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 dot2(f2 ax, f2 ay, f2 az, f2 bx, f2 by, f2 bz)
{
    return fma2(ax, bx, fma2(ay, by, mul2(az, bz)));
}

// system of particle p (of the group's, in ascending order)
__device__ __forceinline__ int pt_system(const PtSys *sys, int nsys, int64_t p)
{
    int lo = 0, hi = nsys;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sys[mid].part0 <= p)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// segment holding index w of an ascending field
template <class F>
__device__ __forceinline__ int pt_find(const PtSeg *seg, int nseg, int64_t w, F field)
{
    int lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (field(seg[mid]) <= w)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int pt_row(int il, int c) { return 6 * (il >> 1) + 2 * c + (il & 1); }

// The three bfloat16 parts of v, as 16-bit patterns: v = h + m + l to 2^-27 of |v|.
__device__ __forceinline__ void split3(double v, unsigned short &h, unsigned short &m, unsigned short &l)
{
    const __nv_bfloat16 bh = __float2bfloat16_rn((float)v);
    const float r1 = (float)(v - (double)__bfloat162float(bh));
    const __nv_bfloat16 bm = __float2bfloat16_rn(r1);
    const __nv_bfloat16 bl = __float2bfloat16_rn(r1 - __bfloat162float(bm));
    h = __bfloat16_as_ushort(bh);
    m = __bfloat16_as_ushort(bm);
    l = __bfloat16_as_ushort(bl);
}

// One block: a row block (42 particles) against 32 particles k (three slabs).  A thread holds one particle
// i and 8 particles k: 24 columns of its three rows, three 16-byte chunks per row and split.  The stores
// are 16-byte pieces that L2 merges: 70 us at n = 2048 (7% of the product's time; 2% at n = 8192).  Laying the
// block's 72 KB out in shared memory and writing them with one bulk copy took 76.5 us.
constexpr int PT_PANEL_THREADS = 192;
template <bool TANGENT>
__global__ void __launch_bounds__(PT_PANEL_THREADS) k_pt_panel(Pos pos, const PtSeg *__restrict__ seg, int nseg,
                                                              unsigned char *__restrict__ panel)
{
    const PtSeg s = seg[pt_find(seg, nseg, (int64_t)blockIdx.x, [](const PtSeg &q) { return (int64_t)q.gen0; })];
    const int groups = s.nslab / 3;
    const int task = (int)blockIdx.x - s.gen0;
    const int rb = task / groups, kg = task - rb * groups;
    const int il = threadIdx.x % 48, oct = threadIdx.x / 48;
    if (il > PT_PART + 1) return;  // 42 and 43 are the two rows left over
    const int i = rb * PT_PART + il;
    const bool row_ok = il < PT_PART && i < s.n;
    double xi = 0.0, yi = 0.0, zi = 0.0, ui = 0.0, vi = 0.0, wi = 0.0;
    if (row_ok) {
        xi = pos.x[s.part0 + i];
        yi = pos.y[s.part0 + i];
        zi = pos.z[s.part0 + i];
        if (TANGENT) {
            ui = pos.dx[s.part0 + i];
            vi = pos.dy[s.part0 + i];
            wi = pos.dz[s.part0 + i];
        }
    }
    // packed bfloat16 pairs of the 24 columns: [split][row a][12 words]
    unsigned int w[3][3][12];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 12; ++c) w[q][a][c] = 0u;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int k = s.k0 + kg * 32 + oct * 8 + e;
        double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // xx xy xz yy yz zz
        if (row_ok && k < s.n && k != i) {
            const double x = pos.x[s.part0 + k] - xi, y = pos.y[s.part0 + k] - yi, z = pos.z[s.part0 + k] - zi;
            const double ri = rsqrt(fma(x, x, fma(y, y, z * z)));
            const double ri2 = ri * ri, i3 = ri * ri2, s5 = 3.0 * i3 * ri2;
            if (TANGENT) {  // dT along the directions: r' = (u v w)
                const double u = pos.dx[s.part0 + k] - ui, v = pos.dy[s.part0 + k] - vi, w = pos.dz[s.part0 + k] - wi;
                const double rr = fma(x, u, fma(y, v, z * w)), c = s5 * rr, e = -5.0 * c * ri2;
                t[0] = fma(e * x, x, fma(2.0 * s5 * x, u, c));
                t[1] = fma(e * x, y, s5 * fma(x, v, y * u));
                t[2] = fma(e * x, z, s5 * fma(x, w, z * u));
                t[3] = fma(e * y, y, fma(2.0 * s5 * y, v, c));
                t[4] = fma(e * y, z, s5 * fma(y, w, z * v));
                t[5] = fma(e * z, z, fma(2.0 * s5 * z, w, c));
            } else {
                t[0] = fma(s5 * x, x, -i3);
                t[1] = s5 * x * y;
                t[2] = s5 * x * z;
                t[3] = fma(s5 * y, y, -i3);
                t[4] = s5 * y * z;
                t[5] = fma(s5 * z, z, -i3);
            }
        }
        constexpr int at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            unsigned short p[3];
            split3(t[c], p[0], p[1], p[2]);
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    if (at[a][b] == c) {
                        const int col = 3 * e + b;
#pragma unroll
                        for (int q = 0; q < 3; ++q) w[q][a][col >> 1] |= (unsigned int)p[q] << ((col & 1) * 16);
                    }
        }
    }
    unsigned char *base = panel + s.mem + ((int64_t)rb * s.nslab + kg * 3) * PT_BLOCK_BYTES;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int row = pt_row(il, a);
        if (row >= PT_ROWS) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int chunk = oct * 3 + c;  // of the group's 12
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                unsigned char *dst = base + (chunk >> 2) * PT_BLOCK_BYTES + q * PT_SPLIT_BYTES + (row >> 3) * 512 +
                                     (chunk & 3) * 128 + (row & 7) * 16;
                *(uint4 *)dst = make_uint4(w[q][a][4 * c], w[q][a][4 * c + 1], w[q][a][4 * c + 2], w[q][a][4 * c + 3]);
            }
        }
    }
}

// Sums of 18 values over the warp's lanes into dst[0 .. 17] (a butterfly that halves the values with the
// lanes: 16, then the last two).
__device__ __forceinline__ void warp_sums18(float *v, float *dst, int lane)
{
#pragma unroll
    for (int o = 16, m = 8; o >= 2; o >>= 1, m >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (q < m) {
                const float keep = up ? v[q + m] : v[q], send = up ? v[q] : v[q + m];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    const bool up = (lane & 16) != 0;
    float w = (up ? v[17] : v[16]) + __shfl_xor_sync(0xffffffffu, up ? v[16] : v[17], 16);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if ((lane & 1) == 0) dst[(lane >> 4 & 1) * 8 + (lane >> 3 & 1) * 4 + (lane >> 2 & 1) * 2 + (lane >> 1 & 1)] = v[0];
    if ((lane & 15) == 0) dst[16 + (lane >> 4)] = w;
}

// One item of a cluster: row blocks 2 a and 2 a + 1 (one per block) and column blocks 2 b and 2 b + 1 of G
// over one segment's k.
struct PtItem {
    PtSeg s;
    int a, b;
};
__device__ __forceinline__ PtItem pt_item(const PtSeg *seg, int nseg, const unsigned int *tiles, int64_t w)
{
    PtItem it;
    it.s = seg[pt_find(seg, nseg, w, [](const PtSeg &q) { return q.item0; })];
    const unsigned int t = tiles[it.s.tab + (w - it.s.item0)];
    it.a = (int)(t >> 16);
    it.b = (int)(t & 0xffffu);
    return it;
}

// MODE 0: forces (and energy).  The adjoint's H d, with T' and r' the rates of T and r along d, is
//   sum_j (G'_ij : dT/dr + G_ij : d(dT/dr)/dr r'),  G' = T' T + T T'
// MODE 1: forces, energy and the second term, from G; MODE 2: the first, from G', whose two products follow
// one another into the same sums (panel2 holds T').
template <int MODE, bool ENERGY>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PT_WARPS * 32, 1)
    k_pt_gemm(Pos pos, const PtSeg *__restrict__ seg, int nseg, int64_t items, const unsigned int *__restrict__ tiles,
              const unsigned char *__restrict__ panel, const unsigned char *__restrict__ panel2,
              double *__restrict__ slots, double *__restrict__ slots2, double nu, PtWait wt)
{
    extern __shared__ __align__(1024) unsigned char smraw[];
    PtShared &S = *(PtShared *)smraw;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto slabs_of = [](const PtItem &it) { return MODE == 2 ? 2 * it.s.nslab : it.s.nslab; };
    const int rank = blockIdx.x & 1, cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        for (int k = 0; k < PT_STAGES; ++k) {
            bar_init(&S.full[k], rank == 0 ? 2 : 1);  // block 0 also waits for block 1's loads
            bar_init(&S.empty[k], 1);
        }
        for (int k = 0; k < 2; ++k) {
            bar_init(&S.acc_full[k], 1);
            bar_init(&S.acc_empty[k], 16);
        }
        bar_init(&S.geo_full, 2);
        bar_init(&S.geo_empty, 8);
        bar_init(&S.drained, 1);
        S.dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&S.tmem))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // both blocks' barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned int tmem = S.tmem;

    // registers: 168 x 384 at launch = 216 x 256 + 72 x 128
    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 8 && lane == 0) {
            unsigned int n = 0;  // slabs loaded
            for (int64_t w = cluster; w < items; w += clusters) {
                const PtItem it = pt_item(seg, nseg, tiles, w);
                const int64_t row = (int64_t)it.s.nslab * PT_BLOCK_BYTES;
                const int64_t oa = it.s.mem + (2 * it.a + rank) * row, ob = it.s.mem + (2 * it.b + rank) * row;
                for (int k = 0; k < slabs_of(it); ++k, ++n) {
                    const int st = n % PT_STAGES;
                    if (!bar_wait(&S.empty[st], ((n / PT_STAGES) & 1) ^ 1, S, wt)) break;
                    // MODE 2: T' T, then T T'
                    const bool second = MODE == 2 && k >= it.s.nslab;
                    const int64_t ko = (int64_t)(second ? k - it.s.nslab : k) * PT_BLOCK_BYTES;
                    unsigned char *dst = S.stage[st];
                    bar_expect(&S.full[st], PT_STAGE_BYTES);
                    bulk_load(dst, (MODE == 2 && !second ? panel2 : panel) + oa + ko, PT_BLOCK_BYTES, &S.full[st]);
                    bulk_load(dst + PT_BLOCK_BYTES, (second ? panel2 : panel) + ob + ko, PT_BLOCK_BYTES, &S.full[st]);
                }
                if (*(volatile int *)&S.dead) break;
            }
            // a block that gave up leaves no copy in flight behind it
            if (*(volatile int *)&S.dead)
                for (unsigned int k = n > PT_STAGES ? n - PT_STAGES : 0; k < n; ++k) {
                    const long long t0 = clock64();
                    while (!bar_try(&S.full[k % PT_STAGES], (k / PT_STAGES) & 1) && clock64() - t0 < 200000000ll) {
                    }
                }
        }
        if (warp == 9 && lane == 0 && rank == 1) {
            // tell block 0, which issues the products of both, that this block's slab is there
            unsigned int n = 0;
            for (int64_t w = cluster; w < items; w += clusters) {
                const PtItem it = pt_item(seg, nseg, tiles, w);
                for (int k = 0; k < slabs_of(it); ++k, ++n) {
                    if (!bar_wait(&S.full[n % PT_STAGES], (n / PT_STAGES) & 1, S, wt)) break;
                    bar_relay_copy(&S.full[n % PT_STAGES], 0);
                }
                if (*(volatile int *)&S.dead) break;
            }
        }
        if (warp == 9 && lane == 0 && rank == 0) {
            unsigned int n = 0;
            bool ok = true;
            for (int64_t w = cluster; ok && w < items; w += clusters) {
                const PtItem it = pt_item(seg, nseg, tiles, w);
                for (int k = 0; k < slabs_of(it); ++k, ++n) {
                    const int st = n % PT_STAGES, buf = n & 1;
                    ok = bar_wait(&S.acc_empty[buf], ((n >> 1) & 1) ^ 1, S, wt) &&
                         bar_wait<true>(&S.full[st], (n / PT_STAGES) & 1, S, wt);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned int A = smem_u32(S.stage[st]), B = A + PT_BLOCK_BYTES, D = tmem + buf * 256;
                    // the small products first (l h, h l, m m, m h, h m), h h last
                    constexpr int qa[6] = {2, 0, 1, 1, 0, 0}, qb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk)
                            mma_bf16(D, operand_desc(A + qa[p] * PT_SPLIT_BYTES + kk * 256),
                                     operand_desc(B + qb[p] * PT_SPLIT_BYTES + kk * 256), p + kk > 0);
                    mma_commit(&S.empty[st]);
                    mma_commit(&S.acc_full[buf]);
                }
            }
            if (!ok) {  // products in flight end before the accumulators are given back
                mma_commit_local(&S.drained);
                const long long t0 = clock64();
                while (!bar_try(&S.drained, 0) && clock64() - t0 < 200000000ll) {
                }
            }
        }
        if (warp >= 10) {
            // the positions of the tile's particles, fetched while its product runs
            unsigned int m = 0;
            for (int64_t w = cluster; w < items; w += clusters, ++m) {
                const PtItem it = pt_item(seg, nseg, tiles, w);
                const int i0 = (2 * it.a + rank) * PT_PART, j0 = 2 * it.b * PT_PART;
                bar_wait(&S.geo_empty, (m & 1) ^ 1, S, wt);
                for (int q = (warp - 10) * 32 + lane; q < 3 * PT_PART; q += 64) {
                    const bool is_j = q < 2 * PT_PART;
                    const int64_t p = it.s.part0 + min(is_j ? j0 + q : i0 + q - 2 * PT_PART, it.s.n - 1);
                    double *d = is_j ? &S.xj[0][q] : &S.xi[0][q - 2 * PT_PART];
                    const int step = is_j ? 2 * PT_PART : PT_PART;
                    d[0] = pos.x[p];
                    d[step] = pos.y[p];
                    d[2 * step] = pos.z[p];
                    if (MODE == 1) {
                        d[3 * step] = pos.dx[p];
                        d[4 * step] = pos.dy[p];
                        d[5 * step] = pos.dz[p];
                    }
                }
                __syncwarp();
                if (lane == 0) bar_arrive(&S.geo_full);
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int quad = warp & 3, half = warp >> 2;
        const int row = quad * 32 + lane, ip = 2 * (row / 6) + (row & 1), al = row % 6 >> 1;
        const f2 ex = pack2(al == 0, al == 0), ey = pack2(al == 1, al == 1), ez = pack2(al == 2, al == 2);  // unit vector
        const f2 m5 = pack2(-5.f, -5.f), c3 = pack2(3.f, 3.f), m1 = pack2(-1.f, -1.f);
        const unsigned int taddr = tmem + ((unsigned int)(quad * 32) << 16) + half * 128;
        unsigned int n = 0, m = 0;
        for (int64_t w = cluster; w < items; w += clusters, ++m) {
            const PtItem it = pt_item(seg, nseg, tiles, w);
            f2 g2[64];  // columns 2 c and 2 c + 1
#pragma unroll
            for (int c = 0; c < 64; ++c) g2[c] = 0ull;
            for (int k = 0; k < slabs_of(it); ++k, ++n) {
                const int buf = n & 1;
                if (!bar_wait(&S.acc_full[buf], (n >> 1) & 1, S, wt)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float t[64];
                    TM_LD64(t, taddr + buf * 256 + c * 64);
                    TM_WAIT64(t);
                    if (c == 1) {  // the accumulator is in registers: free for the next but one slab
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) bar_arrive_tmem(&S.acc_empty[buf], 0);
                    }
#pragma unroll
                    for (int q = 0; q < 32; ++q) g2[c * 32 + q] = add2(g2[c * 32 + q], pack2(t[2 * q], t[2 * q + 1]));
                }
            }
            // G_ii has no part in the results, but T_ij of a pair closer than 4e-7 makes it infinite: the column of the
            // row's own particle is left out as the contraction reads it (in place, ahead of it, the sums' register
            // pairs came apart: 265 M instructions at n = 2048 for 197 M)
            const int self = it.a == it.b && half == rank ? ip : -1;
            auto kept = [&](f2 g, int p) {
                return g & ((f2)(self == 2 * p + 1 ? 0u : ~0u) << 32 | (self == 2 * p ? 0u : ~0u));
            };
            // Geometry of the tile's pairs: n = r / |r| and r^-4, rounded once from FP64 (in FP32 their rounding
            // would count four times in the force).  1 / r is the FP32 approximation t with one step on its
            // FP64 residual, t (1 + (1 - r^2 t^2) / 2): 2^-44.  Done here, in the pause of the product, since
            // the operands' reads leave shared memory no room for it while the product runs.
            const int i0 = (2 * it.a + rank) * PT_PART, j0 = 2 * it.b * PT_PART;
            bar_wait(&S.geo_full, m & 1, S, wt);
            // this warp's sums for the i of its rows, for its energy, and the tile's results from all warps'
            auto store_i = [&](double x, double y, double z) {
                S.fi[half][row][0] = x;
                S.fi[half][row][1] = y;
                S.fi[half][row][2] = z;
            };
            auto store_e = [&](double e) {
                if (!ENERGY) return;
                e = warp_sum(e);
                if (lane == 0) S.e[warp] = e;
            };
            auto write_slot = [&](double *to, bool with_energy) {
                double *slot = to + (it.s.slot0 + (int64_t)it.b * (it.b + 1) + 2 * it.a + rank) * PT_SLOT;
                const int t = threadIdx.x;
                if ((t & 127) < 126) {
                    double v = 0.0;
                    for (int q = 0; q < 4; ++q) v += (double)S.fj[(t >> 7) * 4 + q][t & 127];
                    const int c = t & 127;
                    slot[126 + (t >> 7) * 126 + 3 * (2 * (c / 6) + (c & 1)) + (c % 6 >> 1)] = -nu * v;
                }
                if (t < 126) {
                    const int p = t / 3, c = t - 3 * p;
                    double v = 0.0;
                    for (int h = 0; h < 2; ++h)
                        for (int q = 0; q < 3; ++q) v += S.fi[h][pt_row(p, q)][c];
                    slot[t] = nu * v;
                }
                if (with_energy && t == 255) {
                    double v = 0.0;
                    for (int q = 0; q < 8; ++q) v += S.e[q];
                    slot[378] = -nu * v / 9.0;
                }
            };
            const int go = (MODE == 1 ? 0 : half * (PT_PART / 2) * PT_PART) + (row < 3 * PT_PART ? ip : 0);
            const float rv = row < 3 * PT_PART ? 1.f : 0.f;
            double fx = 0.0, fy = 0.0, fz = 0.0, en = 0.0;
            [[maybe_unused]] double hx = 0.0, hy = 0.0, hz = 0.0;
            if constexpr (MODE == 1) {
                // One column block after the other, since shared memory holds the geometry and its rates for
                // one: all warps form them, the block's four contract.  The rates along d are m = n' (the part
                // of r' across n, over r) and q = |r|' / |r|; with U = y e + n_al g + (g_al - 5 n_al y) n the
                // contraction r^-4 U of the forces has the rate
                //   r^-4 (y' e + m_al g - 5 (m_al y + n_al y') n + (g_al - 5 n_al y) m - 4 q U),  y' = g.m
                constexpr int HALF = PT_GEO / 2;
                float4 *gn = &S.geo[0][0], *gm = gn + 2 * HALF;
                for (int h = 0; h < 2; ++h) {
                    if (h) asm volatile("bar.sync 1, 256;" ::: "memory");  // the first block has been contracted
                    for (int q = threadIdx.x; q < HALF; q += 256) {
                        const int jp = q / PT_PART, il = q - jp * PT_PART, i = i0 + il, jl = h * PT_PART + 2 * jp;
                        float v[2][8];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int j = j0 + jl + u;
                            const double x = S.xj[0][jl + u] - S.xi[0][il], y = S.xj[1][jl + u] - S.xi[1][il],
                                         z = S.xj[2][jl + u] - S.xi[2][il];
                            const double r2 = fma(x, x, fma(y, y, z * z)), t = (double)rsqrt_((float)r2);
                            const double ri = fma(0.5 * fma(-r2, t * t, 1.0), t, t), ri2 = ri * ri;
                            const double nx = x * ri, ny = y * ri, nz = z * ri;
                            const double mx = (S.xj[3][jl + u] - S.xi[3][il]) * ri, my = (S.xj[4][jl + u] - S.xi[4][il]) * ri,
                                         mz = (S.xj[5][jl + u] - S.xi[5][il]) * ri;
                            const double qr = fma(nx, mx, fma(ny, my, nz * mz));
                            const double w[8] = {nx,
                                                 ny,
                                                 nz,
                                                 ri2 * ri2,
                                                 fma(-qr, nx, mx),
                                                 fma(-qr, ny, my),
                                                 fma(-qr, nz, mz),
                                                 -4.0 * qr};
                            const bool ok = i < j && j < it.s.n;
#pragma unroll
                            for (int k = 0; k < 8; ++k) v[u][k] = ok ? (float)w[k] : 0.f;
                        }
                        gn[q] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
                        gn[HALF + q] = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
                        gm[q] = make_float4(v[0][4], v[1][4], v[0][5], v[1][5]);
                        gm[HALF + q] = make_float4(v[0][6], v[1][6], v[0][7], v[1][7]);
                    }
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (h == 1 && lane == 0) bar_arrive(&S.geo_empty);
                    if (half != h) continue;
#pragma unroll
                    for (int p3 = 0; p3 < PT_PART / 2; p3 += 3) {
                        f2 sx = 0ull, sy = 0ull, sz = 0ull, se = 0ull, tx = 0ull, ty = 0ull, tz = 0ull;
                        float fv[18];  // on the j, in the order of the columns
#pragma unroll
                        for (int p = p3; p < p3 + 3; ++p) {
                            const int q = p * PT_PART + go;
                            const float4 A = gn[q], B = gn[HALF + q], C = gm[q], D = gm[HALF + q];
                            const f2 nx = pack2(A.x, A.y), ny = pack2(A.z, A.w), nz = pack2(B.x, B.y);
                            const f2 mx = pack2(C.x, C.y), my = pack2(C.z, C.w), mz = pack2(D.x, D.y), q4 = pack2(D.z, D.w);
                            const f2 i4 = pack2(B.z * rv, B.w * rv);
                            const f2 gx = kept(g2[3 * p], p), gy = kept(g2[3 * p + 1], p), gz = kept(g2[3 * p + 2], p);
                            const f2 y = dot2(gx, gy, gz, nx, ny, nz), yd = dot2(gx, gy, gz, mx, my, mz);
                            const f2 na = al == 0 ? nx : al == 1 ? ny : nz, ga = al == 0 ? gx : al == 1 ? gy : gz,
                                     ma = al == 0 ? mx : al == 1 ? my : mz;
                            const f2 nay = mul2(na, y), sc = fma2(m5, nay, ga), dc = mul2(m5, fma2(ma, y, mul2(na, yd)));
                            const f2 ux = fma2(ex, y, fma2(na, gx, mul2(sc, nx))), uy = fma2(ey, y, fma2(na, gy, mul2(sc, ny))),
                                     uz = fma2(ez, y, fma2(na, gz, mul2(sc, nz)));
                            const f2 vx = mul2(ux, i4), vy = mul2(uy, i4), vz = mul2(uz, i4);
                            sx = add2(sx, vx);
                            sy = add2(sy, vy);
                            sz = add2(sz, vz);
                            const int o = 6 * (p - p3);
                            unpack2(vx, fv[o], fv[o + 1]);
                            unpack2(vy, fv[o + 2], fv[o + 3]);
                            unpack2(vz, fv[o + 4], fv[o + 5]);
                            if (ENERGY) {
                                const float q0 = rsqrt_(fmaxf(B.z, 1e-36f)), q1 = rsqrt_(fmaxf(B.w, 1e-36f));  // r^2
                                se = fma2(mul2(i4, pack2(q0 * rsqrt_(q0), q1 * rsqrt_(q1))), fma2(c3, nay, mul2(m1, ga)), se);
                            }
                            g2[3 * p] = mul2(fma2(ex, yd, fma2(ma, gx, fma2(dc, nx, fma2(sc, mx, mul2(q4, ux))))), i4);
                            g2[3 * p + 1] = mul2(fma2(ey, yd, fma2(ma, gy, fma2(dc, ny, fma2(sc, my, mul2(q4, uy))))), i4);
                            g2[3 * p + 2] = mul2(fma2(ez, yd, fma2(ma, gz, fma2(dc, nz, fma2(sc, mz, mul2(q4, uz))))), i4);
                            tx = add2(tx, g2[3 * p]);
                            ty = add2(ty, g2[3 * p + 1]);
                            tz = add2(tz, g2[3 * p + 2]);
                        }
                        warp_sums18(fv, &S.fj[warp][6 * p3], lane);
                        float u0, u1;
                        unpack2(sx, u0, u1);
                        fx += (double)(u0 + u1);
                        unpack2(sy, u0, u1);
                        fy += (double)(u0 + u1);
                        unpack2(sz, u0, u1);
                        fz += (double)(u0 + u1);
                        unpack2(se, u0, u1);
                        if (ENERGY) en += (double)(u0 + u1);
                        unpack2(tx, u0, u1);
                        hx += (double)(u0 + u1);
                        unpack2(ty, u0, u1);
                        hy += (double)(u0 + u1);
                        unpack2(tz, u0, u1);
                        hz += (double)(u0 + u1);
                    }
                }
                store_i(fx, fy, fz);
                store_e(en);
                asm volatile("bar.sync 1, 256;" ::: "memory");
                write_slot(slots, ENERGY);
                asm volatile("bar.sync 1, 256;" ::: "memory");
                fx = hx;
                fy = hy;
                fz = hz;
            } else {
            for (int q = threadIdx.x; q < PT_GEO; q += 256) {
                const int jp = q / PT_PART, il = q - jp * PT_PART, i = i0 + il;
                const double xi = S.xi[0][il], yi = S.xi[1][il], zi = S.xi[2][il];
                float v[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int j = j0 + 2 * jp + u;
                    const double x = S.xj[0][2 * jp + u] - xi, y = S.xj[1][2 * jp + u] - yi, z = S.xj[2][2 * jp + u] - zi;
                    const double r2 = fma(x, x, fma(y, y, z * z)), t = (double)rsqrt_((float)r2);
                    const double ri = fma(0.5 * fma(-r2, t * t, 1.0), t, t), ri2 = ri * ri;
                    const bool ok = i < j && j < it.s.n;
                    v[u][0] = ok ? (float)(x * ri) : 0.f;
                    v[u][1] = ok ? (float)(y * ri) : 0.f;
                    v[u][2] = ok ? (float)(z * ri) : 0.f;
                    v[u][3] = ok ? (float)(ri2 * ri2) : 0.f;
                }
                S.geo[0][q] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
                S.geo[1][q] = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (lane == 0) bar_arrive(&S.geo_empty);
            // contraction: this thread's row (i, al) of G against dT_ij/dr for the 42 particles j of its
            // column block, two at a time; with g the row of G_ij, n = r / |r|, y = g.n and the unit vector e
            // of the row, its part of G_ij : dT/dr is 3 / r^4 (y e + n_al g + (g_al - 5 n_al y) n)
#pragma unroll
            for (int p3 = 0; p3 < PT_PART / 2; p3 += 3) {
                f2 sx = 0ull, sy = 0ull, sz = 0ull, se = 0ull;
#pragma unroll
                for (int p = p3; p < p3 + 3; ++p) {
                    const float4 A = S.geo[0][go + p * PT_PART], B = S.geo[1][go + p * PT_PART];
                    const f2 nx = pack2(A.x, A.y), ny = pack2(A.z, A.w), nz = pack2(B.x, B.y);
                    const f2 i4 = pack2(B.z * rv, B.w * rv);
                    const f2 gx = kept(g2[3 * p], p), gy = kept(g2[3 * p + 1], p), gz = kept(g2[3 * p + 2], p);
                    const f2 y = dot2(gx, gy, gz, nx, ny, nz);
                    const f2 na = al == 0 ? nx : al == 1 ? ny : nz, ga = al == 0 ? gx : al == 1 ? gy : gz;
                    const f2 nay = mul2(na, y), sc = fma2(m5, nay, ga);
                    const f2 vx = mul2(fma2(ex, y, fma2(na, gx, mul2(sc, nx))), i4);
                    const f2 vy = mul2(fma2(ey, y, fma2(na, gy, mul2(sc, ny))), i4);
                    const f2 vz = mul2(fma2(ez, y, fma2(na, gz, mul2(sc, nz))), i4);
                    sx = add2(sx, vx);
                    sy = add2(sy, vy);
                    sz = add2(sz, vz);
                    if (ENERGY) {  // row al of G_ij : T_ij, with r^-3 = r^-4 r
                        const float q0 = rsqrt_(fmaxf(B.z, 1e-36f)), q1 = rsqrt_(fmaxf(B.w, 1e-36f));  // r^2
                        se = fma2(mul2(i4, pack2(q0 * rsqrt_(q0), q1 * rsqrt_(q1))), fma2(c3, nay, mul2(m1, ga)), se);
                    }
                    g2[3 * p] = vx;
                    g2[3 * p + 1] = vy;
                    g2[3 * p + 2] = vz;
                }
                float u0, u1;
                unpack2(sx, u0, u1);
                fx += (double)(u0 + u1);
                unpack2(sy, u0, u1);
                fy += (double)(u0 + u1);
                unpack2(sz, u0, u1);
                fz += (double)(u0 + u1);
                unpack2(se, u0, u1);
                if (ENERGY) en += (double)(u0 + u1);
            }
            }
            float g[128];
#pragma unroll
            for (int c = 0; c < 63; ++c) unpack2(g2[c], g[2 * c], g[2 * c + 1]);
            g[126] = g[127] = 0.f;
            // f_j: sums over the warp's 32 rows, 4 columns left per lane
#pragma unroll
            for (int o = 16, m = 64; o >= 1; o >>= 1, m >>= 1) {
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int q = 0; q < 64; ++q)
                    if (q < m) {
                        const float keep = up ? g[q + m] : g[q], send = up ? g[q] : g[q + m];
                        g[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
            }
            const int col = ((lane >> 4) & 1) * 64 + ((lane >> 3) & 1) * 32 + ((lane >> 2) & 1) * 16 +
                            ((lane >> 1) & 1) * 8 + (lane & 1) * 4;
            *(float4 *)&S.fj[warp][col] = make_float4(g[0], g[1], g[2], g[3]);
            store_i(fx, fy, fz);
            if (MODE == 0) store_e(en);
            asm volatile("bar.sync 1, 256;" ::: "memory");
            write_slot(MODE == 0 ? slots : slots2, MODE == 0 && ENERGY);
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // no arrival or product of the other block is left
    if (warp == 9)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// ---------------------------------------------------------------------------------------------
// FP64 form.  Only the symmetric part of G_ij acts on the symmetric dT/dr, and sym(T_ik T_kj) is a symmetric
// bilinear form of the two tensors: with A = T_ik, B = T_jk, traceless, its entries are sums of
//   A_xx B_xx, A_yy B_yy, A_zz B_zz, A_xy B_xy, A_xz B_xz, A_yz B_yz                         (d_x d_y d_z, s_xy ..)
// and, since ab' + a'b = (a + b)(a' + b') - aa' - bb', of six products of sums, (A_xy + A_zz)(B_xy + B_zz),
// (A_xz + A_yz)(..), (A_xz + A_yy)(..), (A_xy + A_yz)(..), (A_yz + A_xx)(..), (A_xy + A_xz)(..):
//   G_xx = d_x + s_xy + s_xz,  2 G_xy = -(p_0 - s_xy - d_z) + (p_1 - s_xz - s_yz),  and cyclic.
// So twelve features F of every pair tensor give G by twelve products F F^T: 12 FMA per pair and k, 6 n^3 in
// all, where the AUTA sweep takes about 10 n^3 FP64 operations and NATA's three times that.
//
//   k_p64_panel  the features of a range of k, in the order the matrix instruction's operands are read
//   k_p64_gemm   tiles of 32 x 64 particles (a warp: 16 x 16 pairs x 12 sums) by the FP64 matrix instruction,
//                contracted with dT/dr
//
// Bound: the FP64 rate, which the matrix instruction reaches with few warps (36.9 TFLOP/s with 8 on an SM) and
// few shared-memory reads (half the wavefront slots): 192 registers of sums leave one block of 8 warps an SM.
// n = 4001: 27.2 ms, 31 TFLOP/s of products (25.7 with sums over 512 k and T in plain operations, 2.6 times the
// error).
//
// Accuracy.  The sums are folded into a second set after every 64 k, which waits in TMEM (the block uses no other
// and has no registers left); T and the contraction use powers of r with their rounding errors carried along.
// Relative L2 error of the forces against 80-bit arithmetic, lattices and uniform inputs of 300 .. 4001 particles:
// 3.1e-16 .. 5.3e-16, where plain FP64 sums over triplets have 4.4e-16 .. 6.4e-16 (NATA's) and 8.5e-16 .. 1.4e-14
// (AUTA's).  With sums over 512 k, and T in plain operations, 7.3e-16 .. 1.2e-15.
//
// Plain FMA on 2 x 4 pairs a thread, with three 16-byte reads for 8 FMA, reached 0.41 of the rate (n = 8192:
// 477 ms).
constexpr int P64_PART = 32, P64_K = 8, P64_F = 12, P64_STAGES = 3;
[[maybe_unused]] constexpr int P64_CHUNK = 8;  // panel steps (64 k) of the matrix instruction's sums before they are folded
constexpr int P64_BLOCK = P64_K * P64_F * P64_PART;  // doubles of one row block and 8 k: 24 KB
constexpr int P64_SLOT = pt_slot(P64_PART);

// 1 / r^2 and 1 / r^5 to about one rounding, and r^2: rsqrt with the rounding errors of r^2 and of the powers
// carried along to first order.  In plain operations the power's error alone is 4e-16.
struct P64Radius {
    double r2, i2, i5;
};
__device__ __forceinline__ P64Radius p64_radius(double x, double y, double z)
{
    const double px = x * x, py = y * y, pz = z * z;
    const double s = py + pz, t = s - py, es = (py - (s - t)) + (pz - t);
    const double r2 = px + s, v = r2 - px, er = (px - (r2 - v)) + (s - v);
    // what r^2 lacks
    const double lo = (er + es) + (fma(x, x, -px) + (fma(y, y, -py) + fma(z, z, -pz)));
    const double h = rsqrt(r2), p = r2 * h;
    const double l = 0.5 * h * (fma(-p, h, 1.0) - fma(fma(r2, h, -p), h, lo * h * h));  // 1 / r = h + l
    const double h2 = h * h, e2 = fma(h, h, -h2), h4 = h2 * h2, h5 = h4 * h;
    const double c5 = fma(5.0 * h4, l, fma(h, fma(2.0 * h2, e2, fma(h2, h2, -h4)), fma(h4, h, -h5)));
    return P64Radius{r2, h2 + fma(2.0 * h, l, e2), h5 + c5};
}

struct P64Shared {
    // row block i, two blocks j: [four k][pair of features][8 particles][particle, k][feature], so that the 32
    // lanes' operands, for two features, are 512 consecutive bytes
    double stage[P64_STAGES][3][P64_BLOCK];
    double fi[4][P64_PART][3], fj[2][2 * P64_PART][3], e[8];
    unsigned long long full[P64_STAGES];
    PtItem item;  // in shared memory, since the sums leave few registers
    unsigned int tmem;
    int dead;
};

#if TBMD_PAIRS_MODULE == 2
__global__ void __launch_bounds__(P64_K * P64_PART) k_p64_panel(Pos pos, const PtSeg *__restrict__ seg, int nseg,
                                                              double *__restrict__ panel)
{
    const PtSeg s = seg[pt_find(seg, nseg, (int64_t)blockIdx.x, [](const PtSeg &q) { return (int64_t)q.gen0; })];
    const int task = (int)blockIdx.x - s.gen0, rb = task / s.nslab, kc = task - rb * s.nslab;
    const int il = threadIdx.x & 31, kl = threadIdx.x >> 5;
    const int i = rb * P64_PART + il, k = s.k0 + kc * P64_K + kl;
    double xx = 0.0, xy = 0.0, xz = 0.0, yy = 0.0, yz = 0.0, zz = 0.0;
    if (i < s.n && k < s.n && i != k) {
        const double x = pos.x[s.part0 + k] - pos.x[s.part0 + i], y = pos.y[s.part0 + k] - pos.y[s.part0 + i],
                     z = pos.z[s.part0 + k] - pos.z[s.part0 + i];
        const double i5 = p64_radius(x, y, z).i5, s5 = 3.0 * i5;
        xx = i5 * fma(2.0 * x, x, -fma(y, y, z * z));
        xy = s5 * (x * y);
        xz = s5 * (x * z);
        yy = i5 * fma(2.0 * y, y, -fma(x, x, z * z));
        yz = s5 * (y * z);
        zz = i5 * fma(2.0 * z, z, -fma(x, x, y * y));
    }
    double *dst = panel + s.mem / 8 + ((int64_t)rb * s.nslab + kc) * P64_BLOCK +
                  ((kl >> 2) * (P64_F / 2) * 4 + (il >> 3)) * 64 + ((il & 7) * 4 + (kl & 3)) * 2;
    const double f[P64_F] = {xx, yy, zz, xy, xz, yz, xy + zz, xz + yz, xz + yy, xy + yz, yz + xx, xy + xz};
#pragma unroll
    for (int m = 0; m < P64_F / 2; ++m) *(double2 *)(dst + m * 256) = make_double2(f[2 * m], f[2 * m + 1]);
}
#endif

// D += A B, A 8 x 4 (lane: row lane / 4, column lane % 4), B 4 x 8 (lane: row lane % 4, column lane / 4), D 8 x 8
// (lane: row lane / 4, columns 2 (lane % 4) and + 1)
__device__ __forceinline__ void mma_f64(double &d0, double &d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// twelve doubles of each lane in 24 columns of TMEM
__device__ __forceinline__ void tm_load12(double *v, unsigned int addr)
{
    int w[24];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%24];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%25];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]), "=r"(w[8]),
          "=r"(w[9]), "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15]), "=r"(w[16]),
          "=r"(w[17]), "=r"(w[18]), "=r"(w[19]), "=r"(w[20]), "=r"(w[21]), "=r"(w[22]), "=r"(w[23])
        : "r"(addr), "r"(addr + 16)
        : "memory");
#pragma unroll
    for (int q = 0; q < 12; ++q) v[q] = __hiloint2double(w[2 * q + 1], w[2 * q]);
}
__device__ __forceinline__ void tm_store12(const double *v, unsigned int addr)
{
    int w[24];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
        w[2 * q] = __double2loint(v[q]);
        w[2 * q + 1] = __double2hiint(v[q]);
    }
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%24], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n\t"
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%25], {%16,%17,%18,%19,%20,%21,%22,%23};" ::"r"(w[0]),
        "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]),
        "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]), "r"(w[18]), "r"(w[19]),
        "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(addr), "r"(addr + 16)
        : "memory");
}

template <bool ENERGY>
__global__ void __launch_bounds__(256, 1)
    k_p64_gemm(Pos pos, const PtSeg *__restrict__ seg, int nseg, int64_t items, const unsigned int *__restrict__ tiles,
               const double *__restrict__ panel, double *__restrict__ slots, double nu, PtWait wt)
{
    extern __shared__ __align__(1024) unsigned char smraw[];
    P64Shared &S = *(P64Shared *)smraw;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int iw = warp & 1, jw = warp >> 1, li = lane >> 2, lj = lane & 3;
    if (threadIdx.x == 0) {
        for (int k = 0; k < P64_STAGES; ++k) bar_init(&S.full[k], 1);
        S.dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&S.tmem))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // this warp's part of TMEM: its 32 lanes, half of the columns
    const unsigned int tmem = S.tmem + ((unsigned int)((warp & 3) * 32) << 16) + (warp >> 2) * 256;
    // thread 0 loads, two steps of 8 k ahead of the products and across items
    int64_t lw = blockIdx.x;  // item that is loaded next, its steps left, its blocks i and j
    int left = 0, nslab = 0, oj = 0;
    unsigned int ln = 0;
    const double *src = nullptr;
    auto load = [&](unsigned int st) {
        if (left == 0) {
            if (lw >= items) return;
            const PtItem q = pt_item(seg, nseg, tiles, lw);
            left = nslab = q.s.nslab;
            src = panel + q.s.mem / 8 + (int64_t)q.a * nslab * P64_BLOCK;
            oj = (2 * q.b - q.a) * nslab;
            lw += gridDim.x;
        }
        if (*(volatile int *)&S.dead) return;
        bar_expect(&S.full[st], 3 * P64_BLOCK * 8);
        bulk_load(S.stage[st][0], src, P64_BLOCK * 8, &S.full[st]);
        bulk_load(S.stage[st][1], src + (int64_t)oj * P64_BLOCK, P64_BLOCK * 8, &S.full[st]);
        bulk_load(S.stage[st][2], src + (int64_t)(oj + nslab) * P64_BLOCK, P64_BLOCK * 8, &S.full[st]);
        ++ln;
        src += P64_BLOCK;
        --left;
    };
    if (threadIdx.x == 0)
        for (unsigned int k = 0; k < P64_STAGES; ++k) load(k);
    unsigned int n = 0;
    for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
        if (threadIdx.x == 0) S.item = pt_item(seg, nseg, tiles, w);
        __syncthreads();
        const PtItem &it = S.item;
        const int steps = it.s.nslab;
        for (int k0 = 0; k0 < steps; k0 += P64_CHUNK) {
            double acc[P64_F][2][4];
#pragma unroll
            for (int m = 0; m < P64_F; ++m)
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[m][q >> 2][q & 3] = 0.0;
            const int k1 = min(k0 + P64_CHUNK, steps);
            for (int kc = k0; kc < k1; ++kc, ++n) {
                const unsigned int st = n % P64_STAGES;
                bar_wait(&S.full[st], (n / P64_STAGES) & 1, S, wt);
                const double2 *I = (const double2 *)S.stage[st][0] + iw * 64 + lane,
                              *J = (const double2 *)S.stage[st][1 + (jw >> 1)] + (jw & 1) * 64 + lane;
#pragma unroll 1
                for (int k = 0; k < P64_K / 4; ++k) {
#pragma unroll
                    for (int m = 0; m < P64_F / 2; ++m) {
                        const int o = (k * (P64_F / 2) + m) * 128;
                        const double2 a[2] = {I[o], I[o + 32]}, b[2] = {J[o], J[o + 32]};
#pragma unroll
                        for (int u = 0; u < 2; ++u)
#pragma unroll
                            for (int v = 0; v < 2; ++v) {
                                mma_f64(acc[2 * m][u][2 * v], acc[2 * m][u][2 * v + 1], a[u].x, b[v].x);
                                mma_f64(acc[2 * m + 1][u][2 * v], acc[2 * m + 1][u][2 * v + 1], a[u].y, b[v].y);
                            }
                    }
                }
                __syncthreads();  // the stage has been read
                if (threadIdx.x == 0) load(st);
            }
            __syncwarp();
            // added to the earlier chunks' sums in TMEM, where the contraction finds them a pair at a time
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                double v[P64_F], old[P64_F] = {};
                if (k0) tm_load12(old, tmem + 2 * P64_F * q);
#pragma unroll
                for (int m = 0; m < P64_F; ++m) v[m] = acc[m][q >> 2][q & 3] + old[m];
                tm_store12(v, tmem + 2 * P64_F * q);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        // contraction of G with dT/dr: with h = 2 G r, q = r.h / 2
        //   f_i += nu / r^5 (h + (tr G - 5 q / r^2) r),  E -= nu / (9 r^3) (3 q / r^2 - tr G)
        const int64_t P = it.s.part0;
        const int ia = it.a * P64_PART + iw * 16 + li, jb = 2 * it.b * P64_PART + jw * 16 + lj * 2;
        double fi[2][3] = {}, en = 0.0;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = jb + (v >> 1) * 8 + (v & 1);
            double fj[3] = {};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = ia + u * 8;
                double g[P64_F];
                tm_load12(g, tmem + 2 * P64_F * (4 * u + v));
                if (i < j && j < it.s.n) {
                    const double x = pos.x[P + j] - pos.x[P + i], y = pos.y[P + j] - pos.y[P + i],
                                 z = pos.z[P + j] - pos.z[P + i];
                    const P64Radius r = p64_radius(x, y, z);
                    const double dx = g[0], dy = g[1], dz = g[2], sxy = g[3], sxz = g[4], syz = g[5];
                    const double gxx = dx + sxy + sxz, gyy = dy + sxy + syz, gzz = dz + sxz + syz;
                    // twice the off-diagonal entries
                    const double gxy = (g[7] - sxz - syz) - (g[6] - sxy - dz);
                    const double gxz = (g[9] - sxy - syz) - (g[8] - sxz - dy);
                    const double gyz = (g[11] - sxy - sxz) - (g[10] - syz - dx);
                    const double hx = fma(2.0 * gxx, x, fma(gxy, y, gxz * z)), hy = fma(gxy, x, fma(2.0 * gyy, y, gyz * z)),
                                 hz = fma(gxz, x, fma(gyz, y, 2.0 * gzz * z));
                    const double tr = gxx + gyy + gzz, qq = 0.5 * fma(hx, x, fma(hy, y, hz * z));
                    const double c = nu * r.i5, d = fma(-5.0 * qq, r.i2, tr);
                    const double vx = c * fma(d, x, hx), vy = c * fma(d, y, hy), vz = c * fma(d, z, hz);
                    fi[u][0] += vx;
                    fi[u][1] += vy;
                    fi[u][2] += vz;
                    fj[0] -= vx;
                    fj[1] -= vy;
                    fj[2] -= vz;
                    if (ENERGY) en -= c * r.r2 * fma(3.0 * qq, r.i2, -tr);
                }
                __syncwarp();
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                for (int o = 4; o < 32; o <<= 1) fj[c] += __shfl_xor_sync(0xffffffffu, fj[c], o);
                if (li == 0) S.fj[iw][jw * 16 + lj * 2 + (v >> 1) * 8 + (v & 1)][c] = fj[c];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                for (int o = 1; o < 4; o <<= 1) fi[u][c] += __shfl_xor_sync(0xffffffffu, fi[u][c], o);
                if (lj == 0) S.fi[jw][iw * 16 + li + u * 8][c] = fi[u][c];
            }
        if (ENERGY) {
            en = warp_sum(en);
            if (lane == 0) S.e[warp] = en;
        }
        __syncthreads();
        double *slot = slots + (it.s.slot0 + (int64_t)it.b * (it.b + 1) + it.a) * P64_SLOT;
        for (int t = threadIdx.x; t < 9 * P64_PART; t += 256) {
            double v;
            if (t < 3 * P64_PART) {
                v = S.fi[0][t / 3][t % 3];
                for (int q = 1; q < 4; ++q) v += S.fi[q][t / 3][t % 3];
            } else {
                const int c = t - 3 * P64_PART;
                v = S.fj[0][c / 3][c % 3] + S.fj[1][c / 3][c % 3];
            }
            slot[t] = v;
        }
        if (ENERGY && threadIdx.x == 0) {
            double v = S.e[0];
            for (int q = 1; q < 8; ++q) v += S.e[q];
            slot[9 * P64_PART] = v / 9.0;
        }
        __syncthreads();
    }
    // a block that gave up leaves no copy in flight behind it
    if (threadIdx.x == 0 && *(volatile int *)&S.dead)
        for (unsigned int k = ln > P64_STAGES ? ln - P64_STAGES : 0; k < ln; ++k) {
            const long long t0 = clock64();
            while (!bar_try(&S.full[k % P64_STAGES], (k / P64_STAGES) & 1) && clock64() - t0 < 200000000ll) {
            }
        }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(S.tmem));
}

// Forces from the tiles' results: particle i of row block a sums the tiles (a, b) of its row and the tiles
// (a', a / 2) of its column, over the system's segments.  A warp per particle; the lanes' sums and their
// tree have a fixed order.  A system whose panels did not fit one launch is added up over launches.  A
// launch that gave up gives NaN.
template <int PART>
__global__ void k_pt_reduce(int64_t p0, int64_t n, const PtSys *__restrict__ sys, int nsys, const double *__restrict__ slots, Out out,
                            bool more, const unsigned int *__restrict__ err)
{
    const int64_t p = p0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (p >= p0 + n) return;
    const PtSys s = sys[pt_system(sys, nsys, p)];
    const int i = (int)(p - s.part0), a = i / PART, il = i - a * PART;
    const int b0 = a >> 1, rows = s.nb2 - b0, cols = 2 * b0 + 2, per = s.nb2 * (s.nb2 + 1);
    double f[3] = {0.0, 0.0, 0.0};
    for (int q = lane; q < s.nseg * (rows + cols); q += 32) {
        const int sg = q / (rows + cols), r = q - sg * (rows + cols);
        const int b = r < rows ? b0 + r : b0, ta = r < rows ? a : r - rows;
        const double *src = slots + (s.slot0 + (int64_t)sg * per + (int64_t)b * (b + 1) + ta) * pt_slot(PART) +
                            (r < rows ? 3 * il : 3 * PART * (1 + (a & 1)) + 3 * il);
        f[0] += src[0];
        f[1] += src[1];
        f[2] += src[2];
    }
    const bool bad = *err != 0u;
    for (int c = 0; c < 3; ++c) f[c] = warp_sum(f[c]);
    if (lane == 0) {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        out.fx[p] = bad ? nan : (s.add || more ? out.fx[p] : 0.0) + f[0];
        out.fy[p] = bad ? nan : (s.add || more ? out.fy[p] : 0.0) + f[1];
        out.fz[p] = bad ? nan : (s.add || more ? out.fz[p] : 0.0) + f[2];
    }
}

// Energy of each system: its tiles' energies, a block per system, in a fixed order.  Adds to energy[s]
// (the caller zeroes it).  NaN after a launch that gave up, as the forces.
template <int PART>
__global__ void __launch_bounds__(512) k_pt_energy(const PtSys *__restrict__ sys, const double *__restrict__ slots,
                                                   double *energy, const unsigned int *__restrict__ err)
{
    __shared__ double part[16];
    const PtSys s = sys[blockIdx.x];
    const int64_t total = (int64_t)s.nseg * s.nb2 * (s.nb2 + 1);
    double e = 0.0;
    for (int64_t q = threadIdx.x; q < total; q += 512) e += slots[(s.slot0 + q) * pt_slot(PART) + 9 * PART];
    e = warp_sum(e);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 16; ++k) e += part[k];
        energy[s.index] = *err != 0u ? __longlong_as_double(0x7ff8000000000000ll) : energy[s.index] + e;
    }
}

template <class K>
static cudaError_t pt_shared(K kern, size_t bytes)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
static int64_t pt_particles(const PtPlan &plan, const PtGroup &g)
{
    const PtSys &first = plan.sys[g.sys0], &last = plan.sys[g.sys0 + g.nsys - 1];
    return last.part0 + last.n - first.part0;
}
template <int PART>
static void pt_reduce(const PtPlan &plan, const PtGroup &g, const PtDev &d, const double *slots, Out to, bool more, cudaStream_t st)
{
    const int64_t np = pt_particles(plan, g);
    k_pt_reduce<PART><<<(unsigned)((np + 7) / 8), 256, 0, st>>>(plan.sys[g.sys0].part0, np, d.sys + g.sys0, g.nsys, slots, to,
                                                               more, d.wait.err);
}
template <class K>
static void pt_gemm(K kern, Pos pos, const PtGroup &g, const PtDev &d, double nu, int sms, cudaStream_t st)
{
    const unsigned blocks = 2 * (unsigned)std::min<int64_t>(g.items, sms / 2);
    kern<<<blocks, PT_WARPS * 32, sizeof(PtShared), st>>>(pos, d.segs + g.seg0, g.nsegs, g.items, d.tiles, d.panel, d.panel2,
                                                         d.slots, d.slots2, nu, d.wait);
}

#if TBMD_PAIRS_MODULE == 1
cudaError_t pt_init_adjoint(bool energy)
{
    const cudaError_t e = pt_shared(energy ? k_pt_gemm<1, true> : k_pt_gemm<1, false>, sizeof(PtShared));
    return e != cudaSuccess ? e : pt_shared(k_pt_gemm<2, false>, sizeof(PtShared));
}

void pt_launch_adjoint(bool second, Pos pos, const PtGroup &g, const PtDev &d, bool energy, double nu, int sms, cudaStream_t st)
{
    if (second) return pt_gemm(k_pt_gemm<2, false>, pos, g, d, nu, sms, st);
    k_pt_panel<true><<<(unsigned)g.gen, PT_PANEL_THREADS, 0, st>>>(pos, d.segs + g.seg0, g.nsegs, d.panel2);
    pt_gemm(energy ? k_pt_gemm<1, true> : k_pt_gemm<1, false>, pos, g, d, nu, sms, st);
}
#elif TBMD_PAIRS_MODULE == 2
cudaError_t pt_init_fp64(bool energy) { return pt_shared(energy ? k_p64_gemm<true> : k_p64_gemm<false>, sizeof(P64Shared)); }

void pt_launch_fp64(Pos pos, Out out, const PtPlan &plan, const PtGroup &g, const PtDev &d, double *energy, double nu,
                    int sms, cudaStream_t st)
{
    const PtSeg *seg = d.segs + g.seg0;
    k_p64_panel<<<(unsigned)g.gen, P64_K * P64_PART, 0, st>>>(pos, seg, g.nsegs, (double *)d.panel);
    auto gemm = energy ? k_p64_gemm<true> : k_p64_gemm<false>;
    gemm<<<(unsigned)std::min<int64_t>(g.items, sms), 256, sizeof(P64Shared), st>>>(
        pos, seg, g.nsegs, g.items, d.tiles, (const double *)d.panel, d.slots, nu, d.wait);
    pt_reduce<P64_PART>(plan, g, d, d.slots, out, false, st);
    if (energy) k_pt_energy<P64_PART><<<(unsigned)g.nsys, 512, 0, st>>>(d.sys + g.sys0, d.slots, energy, d.wait.err);
}
#else
// ---------------------------------------------------------------------------------------------
// Work lists (host)

// Tile order of nb2 column blocks: strips of 8 of them, walked row by row, so that the tiles in flight share
// row and column blocks in L2 (mixed form, one tile per two SMs, rows as wide as columns: 17 blocks, 40 MB
// at 512 k; FP64 form, one per SM, rows half as wide: 53 MB).
static void pt_tiles(int nb2, bool fp64, std::vector<unsigned int> &out)
{
    const int per = fp64 ? 2 : 1;  // rows per column block
    for (int b0 = 0; b0 < nb2; b0 += 8) {
        const int b1 = std::min(nb2, b0 + 8);
        for (int a = 0; a < per * b1; ++a)
            for (int b = std::max(b0, a / per); b < b1; ++b) out.push_back((unsigned int)a << 16 | (unsigned int)b);
    }
}

static int pt_width(bool fp64) { return 2 * (fp64 ? P64_PART : PT_PART); }
static int64_t pt_items(int64_t nb2, bool fp64) { return fp64 ? nb2 * (nb2 + 1) : nb2 * (nb2 + 1) / 2; }
// panel steps of a range of k: slabs of 32 columns (three per 32 particles), or 8 particles
static int pt_steps(int64_t k, bool fp64) { return fp64 ? (int)((k + P64_K - 1) / P64_K) : (int)((k + 31) / 32 * 3); }

// Time in cycles of a launch over ranges of kp particles: the most that one block is dealt (block b takes items
// b, b + units, ... of all ranges in turn).  Mixed: 1,536 cycles a slab (what its product takes) and 14,000 an
// item, while the product pauses (geometry 5,800, contraction 4,800, the rest sums over rows and set-up).  FP64:
// 3,200 cycles for 8 k (3,072 of products), 9,000 an item.  Above 32 items a block the average is as good and much cheaper.
static double pt_cycles(const int64_t *sys_off, int nsys, int units, bool fp64, int kp)
{
    const double step = fp64 ? 3200.0 : 1536.0, item = fp64 ? 9000.0 : 14000.0;
    int64_t items = 0;
    double steps = 0.0;
    for (int s = 0; s < nsys; ++s) {
        const int64_t n = sys_off[s + 1] - sys_off[s], tiles = pt_items((n + pt_width(fp64) - 1) / pt_width(fp64), fp64);
        items += tiles * ((n + kp - 1) / kp);
        steps += (double)tiles * (double)pt_steps(n, fp64);
    }
    if (items > 32 * (int64_t)units)
        return (double)((items + units - 1) / units) * (steps / (double)items * step + item);
    std::vector<double> load((size_t)units, 0.0);
    double every = 0.0;  // of the ranges' whole turns
    int64_t at = 0;
    for (int s = 0; s < nsys; ++s) {
        const int64_t n = sys_off[s + 1] - sys_off[s], tiles = pt_items((n + pt_width(fp64) - 1) / pt_width(fp64), fp64);
        for (int64_t k0 = 0; k0 < n; k0 += kp) {
            const double t = pt_steps(std::min<int64_t>(kp, n - k0), fp64) * step + item;
            every += (double)(tiles / units) * t;
            for (int64_t q = 0; q < tiles % units; ++q) load[(size_t)((at + q) % units)] += t;
            at = (at + tiles) % units;
        }
    }
    return every + *std::max_element(load.begin(), load.end());
}

// Particles k of one item: the range length with the least time, of round lengths and of even splits of the
// largest system, a longer one where it is within 2% (fewer results to store and add).  An estimate from the
// average item does not see a short last range: it took 384 + 128 for n = 512 (all kernels of a call, FP64 121
// us, with 256 + 256 93; mixed 77 and 67; n = 600: 177 and 156, 93 and 77.5).  512 at most, for the accuracy of
// the mixed form's FP32 sums over a range, and for L2.
static int pt_range(const int64_t *sys_off, int nsys, int sms, bool fp64, int most)
{
    const int units = std::max(1, fp64 ? sms : sms / 2);  // items in flight
    int64_t nmax = 1;
    for (int s = 0; s < nsys; ++s) nmax = std::max(nmax, sys_off[s + 1] - sys_off[s]);
    std::vector<int> lengths{512, 384, 256, 192, 128, 96, 64, 32};
    for (int64_t parts = 1; parts <= 8; ++parts)
        lengths.push_back((int)std::min<int64_t>(most, ((nmax + parts - 1) / parts + 31) / 32 * 32));
    std::sort(lengths.begin(), lengths.end(), [](int a, int b) { return a > b; });
    int best = 0, last = 0;
    double least = 0.0;
    for (int kp : lengths) {
        // lengths that no system reaches are the same plan: tried once, since batches of small systems, whose sizes
        // change from call to call, wait for this (200 of 24 particles: 53 -> 9 us, 68 -> 10 in FP64)
        if (kp > most || kp == last || (kp >= nmax && last)) continue;
        last = kp;
        const double t = pt_cycles(sys_off, nsys, units, fp64, kp);
        if (!best || t < 0.98 * least) {
            least = t;
            best = kp;
        }
    }
    return best;
}

// Panels, tiles and results of all systems, in groups whose panel and results stay within `budget` bytes
// (a group has at least one range); a system may go over several groups.
void pt_plan(const int64_t *sys_off, int nsys, int sms, size_t budget, bool fp64, bool dual, PtPlan &plan)
{
    static_assert(P64_BLOCK * sizeof(double) == PT_BLOCK_BYTES, "both forms' panels are planned alike");
    plan = PtPlan{};
    plan.fp64 = fp64;
    plan.slot_bytes = sizeof(double) * (size_t)(fp64 ? P64_SLOT : PT_SLOT);
    const int kp = pt_range(sys_off, nsys, sms, fp64, dual ? 256 : 512);  // G' sums a range twice
    PtGroup g{};
    for (int s = 0; s < nsys; ++s) {
        const int64_t n = sys_off[s + 1] - sys_off[s];
        if (n < 1) continue;
        const int nb2 = (int)((n + pt_width(fp64) - 1) / pt_width(fp64));
        const int64_t tiles = (int64_t)nb2 * (nb2 + 1);
        const int tab = (int)plan.tiles.size();
        pt_tiles(nb2, fp64, plan.tiles);
        PtSys sy{sys_off[s], g.slots, (int)n, nb2, 0, s, 0, 0};
        auto end_system = [&]() {
            if (!sy.nseg) return;
            plan.sys.push_back(sy);
            ++g.nsys;
        };
        for (int64_t k0 = 0; k0 < n; k0 += kp) {
            const int nslab = pt_steps(std::min<int64_t>(kp, n - k0), fp64);
            const size_t mem = (size_t)nb2 * 2 * nslab * PT_BLOCK_BYTES;
            if (g.nsegs && g.mem + mem + (size_t)(g.slots + tiles) * plan.slot_bytes > budget) {
                end_system();
                plan.groups.push_back(g);
                g = PtGroup{};
                g.seg0 = (int)plan.segs.size();
                g.sys0 = (int)plan.sys.size();
                sy.slot0 = 0;
                sy.add = k0 > 0;
                sy.nseg = 0;
            }
            plan.segs.push_back(PtSeg{(int64_t)g.mem, g.items, g.slots, (int)sys_off[s], (int)n, (int)k0, nslab, tab,
                                      g.gen});
            g.mem += mem;
            g.items += pt_items(nb2, fp64);
            g.slots += tiles;
            g.gen += 2 * nb2 * (fp64 ? nslab : nslab / 3);
            ++g.nsegs;
            ++sy.nseg;
        }
        end_system();
    }
    if (g.nsegs) plan.groups.push_back(g);
    for (const PtGroup &q : plan.groups) {
        plan.mem = std::max(plan.mem, q.mem);
        plan.slots = std::max(plan.slots, (size_t)q.slots);
    }
}

// Shared memory of the kernels of one form.  Only those that will run: setting it loads a kernel.
cudaError_t pt_init(bool fp64, bool dual, bool energy)
{
    if (fp64) return pt_init_fp64(energy);
    if (dual) return pt_init_adjoint(energy);
    return pt_shared(energy ? k_pt_gemm<0, true> : k_pt_gemm<0, false>, sizeof(PtShared));
}

// What the tensor core's truncation takes off a product on average.  A truncation loses half an ulp, which is
// 2^-24 / (2 ln 2) = 4.3e-8 of a value with a log-uniform mantissa; a slab's sum is truncated twice at full size, by
// the two hh steps, of which the first holds half of it.  The results' scale makes up for it.  Energies of thermal
// lattices, 130 .. 4000 particles: -6.5e-8 .. -7.5e-8 in every one without (the FP32 sweeps: -2e-8 .. -5e-8).
constexpr double PT_TRUNCATED = 1.5 * 5.9604644775390625e-08 * 0.72134752044448170;

cudaError_t launch_pairs(bool dual, Pos pos, Out out, const PtPlan &plan, const PtDev &d, double *energy,
                         double nu, int sms, cudaStream_t st, int *launches)
{
    static_assert(sizeof(PtShared) <= 232448 && sizeof(P64Shared) <= 232448, "shared memory of one block");
    if (!plan.fp64) nu *= 1.0 + PT_TRUNCATED;
    const Out h{out.hx, out.hy, out.hz, nullptr, nullptr, nullptr};
    for (const PtGroup &g : plan.groups) {
        *launches += energy ? 4 : 3;
        if (plan.fp64) {
            pt_launch_fp64(pos, out, plan, g, d, energy, nu, sms, st);
            continue;
        }
        k_pt_panel<false><<<(unsigned)g.gen, PT_PANEL_THREADS, 0, st>>>(pos, d.segs + g.seg0, g.nsegs, d.panel);
        if (dual) {
            pt_launch_adjoint(false, pos, g, d, energy != nullptr, nu, sms, st);
            pt_reduce<PT_PART>(plan, g, d, d.slots2, h, false, st);
            pt_launch_adjoint(true, pos, g, d, energy != nullptr, nu, sms, st);
            pt_reduce<PT_PART>(plan, g, d, d.slots2, h, true, st);
            *launches += 4;
        } else {
            pt_gemm(energy ? k_pt_gemm<0, true> : k_pt_gemm<0, false>, pos, g, d, nu, sms, st);
        }
        pt_reduce<PT_PART>(plan, g, d, d.slots, out, false, st);
        if (energy) k_pt_energy<PT_PART><<<(unsigned)g.nsys, 512, 0, st>>>(d.sys + g.sys0, d.slots, energy, d.wait.err);
    }
    return cudaGetLastError();
}
#endif

}  // namespace tbmd
