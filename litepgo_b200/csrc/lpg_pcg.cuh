// lpg_pcg.cuh -- block-Jacobi PCG of a whole solve in one cooperative launch, for meshes whose rows fit
// one sliced-ELL chunk per warp (16 per block, one block per SM). Included by lpg_solve.cu, whose vector
// helpers and PcgState it uses.
//
// The launch-per-step iteration (spmv_sell and pcg_update in a graph) is bound at these sizes by its two
// launches and its chain of gathers and reductions through L2. Here a lane keeps its row's x, r, z, p and
// preconditioner block in registers for the whole solve, and a block its chunks' matrix values as far as
// they fit (both triangles, borrowed blocks transposed once): the first slots of a warp in registers, up to
// 16 more in shared memory, the rest read from L2. What crosses blocks is z and three sums:
// - z = D r of the block's rows goes to L2 for the blocks that have it as a neighbour (their halo), which form
//   p = z + beta p of the halo themselves, bit by bit as its owner does; p of both is in shared memory. A
//   vertex's z is one 16-byte word (two in FP64) that carries the iteration's number, so a reader polls the
//   word itself: no fence, no flag, one L2 round trip.
// - The sums r.z and r.r of a block travel at the same time as z, then p.Ap: published as numbered words too;
//   warps of every block poll all of them and add them in block order, so that all blocks hold bitwise the
//   same sums and results do not depend on scheduling.
// Every block has read what an exchange brings before it publishes in the next one, and a word is rewritten
// only after a whole exchange in between: one copy of each suffices. An iteration is then two L2 round trips,
// the products and FP64 latency.
//
// The recurrences are those of the launches per step. The form with one reduction (Chronopoulos and Gear,
// 1989), which takes p.Ap from z.Az and the sums before and A p from a recurrence, saves the second exchange of
// sums (nothing to speak of where a system is on few blocks: pcg_chunks) and is not stable enough in FP32: on
// blocks with a Poisson ratio of 0.4999 it took 60 % more iterations, from 0.499975 on it lost the sign of p.Ap,
// and so it did on columns of 60 cubes.
//
// A batch of meshes is one launch too: every mesh has blocks of its own (one block exchanges nothing), its
// own sums, tolerance and end, where the launches per step run all meshes in lockstep to the slowest.
//
// Measured per iteration, B200 (launch-per-step, then this kernel): 648 vertices FP64 14.2 and 4.0 us; 4,896
// FP64 16.4 and 5.4; 62,197 FP32 15.6 and 7.5, where the products (18 slots a lane) and the wait for the
// slowest block are half; 48 boxes of 4 to 16 cubes, 64,000 vertices, 24 in lockstep and 9.4 side by side. Large
// systems keep three slots of a lane in registers in FP32 (KR), which spills 56 bytes: with two the slowest block
// waits for one more slot from L2 (a Newton solve of 62,197 vertices 90 ms instead of 82), with four the spills cost
// more (86). Beside 227 KB of shared memory there is hardly any L1 to hold them, hence G and one word per lane.
#pragma once

namespace lpg {
namespace {

constexpr int kPcgThreads = 512, kPcgWarps = kPcgThreads / 32;
constexpr int kPcgMaxBlocks = 160; // two sums of five groups of 32 blocks: a polling warp each

// One linear system of a launch: a mesh's chunks and vertices (a chunk at a mesh's ends may hold rows of its
// neighbours, which are passed over) and the blocks that work on it. Groups know nothing of one another.
struct PcgGroup {
    int c0, c1, v0, v1; // chunks and vertices
    int b0, blocks;
};
// Plan of the launch. A block keeps z of its own rows (32 per chunk, in the chunks' order), then of the other
// vertices that are columns of them (its halo, ascending); every slot of the sliced ELL has its column's
// position in that list (indexed as sell_col and sell_bref).
struct PcgPlan {
    const PcgGroup* groups = nullptr;
    const int32_t* of_block = nullptr;   // group of each block
    int halo_stride = 0, blocks = 0;
    const int32_t* halo = nullptr;       // [blocks][halo_stride]
    const int32_t* halo_count = nullptr; // [blocks]
    const uint16_t* idx_own = nullptr;
    const uint16_t* idx_bor = nullptr;
};
__host__ __device__ inline int pcg_first_chunk(const PcgGroup& g, int rank) {
    return g.c0 + static_cast<int>(static_cast<int64_t>(g.c1 - g.c0) * rank / g.blocks);
}

// Position of every vertex in the sliced-ELL row order.
__global__ void row_position_kernel(const DevMesh m, int32_t* pos) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 32 * m.n_sell && m.sell_row[i] >= 0) pos[m.sell_row[i]] = i;
}

// One block per block of the plan: marks the other vertices that its rows refer to in a bitmap over the
// group's vertices, numbers them in ascending order and writes the list (when halo is not null) and the
// slots' positions.
__global__ void __launch_bounds__(kPcgThreads)
    pcg_plan_kernel(const DevMesh m, const PcgGroup* groups, const int32_t* of_block, const int32_t* pos, int32_t* halo,
                    int stride, int32_t* count, uint16_t* idx_own, uint16_t* idx_bor) {
    extern __shared__ unsigned s_bits[]; // bitmap, then the number of marks before each word
    const PcgGroup g = groups[of_block[blockIdx.x]];
    const int words = (g.v1 - g.v0 + 31) / 32;
    unsigned* before = s_bits + words;
    __shared__ unsigned s_sum[kPcgWarps];
    __shared__ unsigned s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < words; i += kPcgThreads) s_bits[i] = 0;
    if (tid == 0) s_base = 0;
    __syncthreads();
    const int rank = blockIdx.x - g.b0, c0 = pcg_first_chunk(g, rank), c1 = pcg_first_chunk(g, rank + 1);
    const int p0 = 32 * c0, p1 = 32 * c1;
    const auto each_slot = [&](auto&& own, auto&& bor) {
        for (int c = c0 + warp; c < c1; c += kPcgWarps) {
            const int row = m.sell_row[32 * static_cast<size_t>(c) + lane];
            if (row < g.v0 || row >= g.v1) continue;
            for (int i = m.sell_ptr[c] + lane; i < m.sell_ptr[c + 1]; i += 32) own(i, m.sell_col[i]);
            for (int i = m.sell_bptr[c] + lane; i < m.sell_bptr[c + 1]; i += 32) bor(i, m.sell_bref[i].y);
        }
    };
    const auto mark = [&](int, int v) {
        if (pos[v] < p0 || pos[v] >= p1) atomicOr(s_bits + ((v - g.v0) >> 5), 1u << ((v - g.v0) & 31));
    };
    each_slot(mark, mark);
    __syncthreads();
    for (int i0 = 0; i0 < words; i0 += kPcgThreads) { // exclusive prefix sums of the words' counts
        const int i = i0 + tid;
        const unsigned n = i < words ? __popc(s_bits[i]) : 0;
        unsigned inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_sum[warp] = inc;
        __syncthreads();
        unsigned pre = s_base;
        for (int w = 0; w < warp; ++w) pre += s_sum[w];
        if (i < words) before[i] = pre + inc - n;
        __syncthreads();
        if (tid == kPcgThreads - 1) s_base = pre + inc;
        __syncthreads();
    }
    if (tid == 0) count[blockIdx.x] = static_cast<int32_t>(s_base);
    if (halo == nullptr) return;
    for (int i = tid; i < words; i += kPcgThreads) {
        unsigned b = s_bits[i], at = before[i];
        for (; b; b &= b - 1) halo[static_cast<size_t>(stride) * blockIdx.x + at++] = g.v0 + 32 * i + __ffs(b) - 1;
    }
    const auto at = [&](int v) {
        if (pos[v] >= p0 && pos[v] < p1) return static_cast<uint16_t>(pos[v] - p0);
        const int w = (v - g.v0) >> 5, bit = (v - g.v0) & 31;
        return static_cast<uint16_t>(p1 - p0 + before[w] + __popc(s_bits[w] & ((1u << bit) - 1u)));
    };
    each_slot([&](int i, int v) { idx_own[i] = at(v); }, [&](int i, int v) { idx_bor[i] = at(v); });
}

// 16-byte words that carry their own validity: single 128-bit accesses, so a reader that finds the number
// it waits for has the rest of the word too, and nothing else orders the two sides.
__device__ __forceinline__ void st_word(void* p, unsigned a, unsigned b, unsigned c, unsigned number) {
    asm volatile("{\n\t.reg .b64 l, h;\n\t.reg .b128 w;\n\tmov.b64 l, {%1, %2};\n\tmov.b64 h, {%3, %4};\n\t"
                 "mov.b128 w, {l, h};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(number)
                 : "memory");
}
__device__ __forceinline__ uint4 ld_word(const void* p) {
    uint4 v;
    asm volatile("{\n\t.reg .b64 l, h;\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%4];\n\tmov.b128 {l, h}, w;\n\t"
                 "mov.b64 {%0, %1}, l;\n\tmov.b64 {%2, %3}, h;\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
// A vertex's z as one word (FP32) or two (FP64), 4 values of R apart.
__device__ __forceinline__ void publish3(float* p, const float z[3], unsigned number) {
    st_word(p, __float_as_uint(z[0]), __float_as_uint(z[1]), __float_as_uint(z[2]), number);
}
__device__ __forceinline__ void publish3(double* p, const double z[3], unsigned number) {
    st_word(p, __double2loint(z[0]), __double2hiint(z[0]), __double2loint(z[1]), number);
    st_word(p + 2, __double2hiint(z[1]), __double2loint(z[2]), __double2hiint(z[2]), number);
}
template <typename R> struct Pending; // the words of one vertex as loaded
template <> struct Pending<float> {
    uint4 a;
    __device__ __forceinline__ void load(const float* p) { a = ld_word(p); }
    __device__ __forceinline__ bool ready(unsigned number) const { return a.w == number; }
    __device__ __forceinline__ void get(float z[3]) const {
        z[0] = __uint_as_float(a.x), z[1] = __uint_as_float(a.y), z[2] = __uint_as_float(a.z);
    }
};
template <> struct Pending<double> {
    uint4 a, b;
    __device__ __forceinline__ void load(const double* p) { a = ld_word(p), b = ld_word(p + 2); }
    __device__ __forceinline__ bool ready(unsigned number) const { return a.w == number && b.w == number; }
    __device__ __forceinline__ void get(double z[3]) const {
        z[0] = __hiloint2double(a.y, a.x), z[1] = __hiloint2double(b.x, a.z), z[2] = __hiloint2double(b.z, b.y);
    }
};

// Values per vertex of p in shared memory: float4 in FP32, three doubles in FP64.
template <typename R> constexpr int pcg_stride() { return sizeof(R) == 4 ? 4 : 3; }
// Shared memory of the split rows' parts, which the halo's z is staged in as it arrives (3 values a vertex).
template <typename R> constexpr size_t pcg_stage_bytes(int halo) {
    constexpr size_t parts = 3 * 32 * kPcgWarps * sizeof(R);
    const size_t z = (3 * halo * sizeof(R) + 15) / 16 * 16;
    return z > parts ? z : parts;
}
// Shared memory of p (own rows and halo), of the halo's vertex list and of the parts.
template <typename R> constexpr size_t pcg_p_bytes(int rows, int halo, bool staged) {
    return (static_cast<size_t>(rows + halo) * pcg_stride<R>() * sizeof(R) + halo * sizeof(int32_t) + 15) / 16 * 16 +
           pcg_stage_bytes<R>(staged ? halo : 0);
}
// Slots of a warp in registers: KR of the kernel, which has two builds. Large systems, whose blocks read values from
// L2, gain more from one more slot on the chip (and in FP32 from three words of the halo in flight) than its
// spills cost; the others run better without. Newton, small build then large: 8^3 cubes mixed 11.4 and 12.4 ms,
// 24^3 FP64 45.6 and 43.6, 36^3 FP64 150 and 134.
template <typename R> constexpr int pcg_register_slots(bool large) { return (sizeof(R) == 4 ? 2 : 1) + (large ? 1 : 0); }
// Warps that share a chunk in a block of nc chunks.
__host__ __device__ constexpr int pcg_sub(int nc) { return 4 * nc <= kPcgWarps ? 4 : 2 * nc <= kPcgWarps ? 2 : 1; }
// Shared memory of one slot of a chunk (32 blocks).
template <typename R> constexpr size_t pcg_slot_bytes() { return 32 * 9 * sizeof(R); }
constexpr size_t kPcgFixed = (2 * kPcgWarps + 22) * sizeof(double); // sums and scalars

template <typename R> struct PcgArgs {
    const R *val, *dinv, *mask4, *b4;
    R *x4, *z4;
    PcgState* st;     // per group, zero before the launch
    uint4* words;     // [3][blocks of the plan]
    unsigned* number; // per group: exchanges so far
    const double* tols; // per group, or null: tol
    const int* act;     // per group (0: x = 0 and nothing else), or null
    double tol;
    int max_iters;
    unsigned polls;         // of one word before the block gives up
    int first_block;        // the plan's first block of this launch
    bool first_direction;   // on negative curvature at the first step, x is the preconditioned residual
    size_t smem;
};

// A staged vertex: one 16-byte access in FP32.
__device__ __forceinline__ void lds3(const float* p, float v[3]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z;
}
__device__ __forceinline__ void lds3(const double* p, double v[3]) { v[0] = p[0], v[1] = p[1], v[2] = p[2]; }
__device__ __forceinline__ void sts3(float* p, const float v[3]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], 0.f);
}
__device__ __forceinline__ void sts3(double* p, const double v[3]) { p[0] = v[0], p[1] = v[1], p[2] = v[2]; }

// A resident slot keeps the lanes' entries 0-3 and 4-7 (FP32; pairs in FP64) as 16-byte accesses, each
// contiguous over the warp, then entry 8.
__device__ __forceinline__ void store_block(float* slot, int lane, const float k[9]) {
    float4* v = reinterpret_cast<float4*>(slot);
    v[lane] = make_float4(k[0], k[1], k[2], k[3]);
    v[32 + lane] = make_float4(k[4], k[5], k[6], k[7]);
    slot[256 + lane] = k[8];
}
__device__ __forceinline__ void load_block(const float* slot, int lane, float k[9]) {
    const float4* v = reinterpret_cast<const float4*>(slot);
    const float4 a = v[lane], b = v[32 + lane];
    k[0] = a.x, k[1] = a.y, k[2] = a.z, k[3] = a.w, k[4] = b.x, k[5] = b.y, k[6] = b.z, k[7] = b.w;
    k[8] = slot[256 + lane];
}
__device__ __forceinline__ void store_block(double* slot, int lane, const double k[9]) {
    double2* v = reinterpret_cast<double2*>(slot);
#pragma unroll
    for (int t = 0; t < 4; ++t) v[32 * t + lane] = make_double2(k[2 * t], k[2 * t + 1]);
    slot[256 + lane] = k[8];
}
__device__ __forceinline__ void load_block(const double* slot, int lane, double k[9]) {
    const double2* v = reinterpret_cast<const double2*>(slot);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const double2 a = v[32 * t + lane];
        k[2 * t] = a.x, k[2 * t + 1] = a.y;
    }
    k[8] = slot[256 + lane];
}

__device__ __forceinline__ double shfl_xor_add(double keep, double send, int o) {
    return keep + __shfl_xor_sync(0xffffffffu, send, o);
}

template <typename R, int KR>
__global__ void __launch_bounds__(kPcgThreads, 1) pcg_solve_kernel(const DevMesh m, const PcgPlan plan, const PcgArgs<R> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int PS = pcg_stride<R>(), G = KR == 3 ? 3 : 1;
    constexpr int MS = 16; // most slots of a warp in shared memory (their column indices are in registers)
    double* red = reinterpret_cast<double*>(smem_raw); // [2 values][warps]
    double* total = red + 2 * kPcgWarps; // [warp]: the sums of 32 blocks
    volatile int* s_lost = reinterpret_cast<volatile int*>(total + 16);
    double* scal = total + 18; // 1 / (r.z of the iteration before), the squared tolerance, |b|^2
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int block = a.first_block + blockIdx.x, grp = plan.of_block[block];
    const PcgGroup g = plan.groups[grp];
    const int blocks = g.blocks, rank = block - g.b0;
    const int c0 = pcg_first_chunk(g, rank), c1 = pcg_first_chunk(g, rank + 1);
    const int nc = c1 - c0; // at most kPcgWarps
    const auto row_of = [&](int c) { // the lane's row, -1 past the end or in another mesh
        const int row = m.sell_row[32 * static_cast<size_t>(c) + lane];
        return row >= g.v0 && row < g.v1 ? row : -1;
    };
    if (a.act != nullptr && a.act[grp] == 0) { // the whole group leaves
        const int row = warp < nc ? row_of(c0 + warp) : -1;
        if (row >= 0) st4(a.x4 + 4 * static_cast<size_t>(row), R(0), R(0), R(0));
        return;
    }
    const int L = plan.halo_count[block], own_rows = 32 * nc;
    const bool staged = kPcgFixed + pcg_p_bytes<R>(own_rows, L, true) <= a.smem;
    R* parts = reinterpret_cast<R*>(smem_raw + kPcgFixed); // [warp][3][32], or the halo's z [L][3]
    R* ps = reinterpret_cast<R*>(smem_raw + kPcgFixed + pcg_stage_bytes<R>(staged ? L : 0));
    int32_t* list = reinterpret_cast<int32_t*>(ps + static_cast<size_t>(PS) * (own_rows + L));
    const size_t vectors = kPcgFixed + pcg_p_bytes<R>(own_rows, L, staged);
    unsigned char* rest = smem_raw + vectors;
    // `sub` warps share a chunk (its slots dealt round robin); the first of them owns the rows.
    const int sub = pcg_sub(nc);
    const int ch = warp / sub, part = warp - sub * ch;
    const bool on = ch < nc;
    const int c = c0 + (on ? ch : 0);
    const int lane_row = row_of(c); // of every warp that shares the chunk
    unsigned free = lane_row >= 0 ? 8u : 0u; // bit 3: the lane has a row; bit i: its component i is free
    const int s0 = m.sell_ptr[c], w0 = (m.sell_ptr[c + 1] - s0) >> 5;
    const int t0 = m.sell_bptr[c], bw = (m.sell_bptr[c + 1] - t0) >> 5;
    const int ns = on ? w0 + bw : 0;
    // Of a chunk's slots (own, then borrowed) the first KR of each of its warps are in registers, as many
    // more as fit are in shared memory (at most `cap` per chunk, the largest cap that fits all chunks: the
    // same walk in every thread), the rest are read from L2.
    const auto slots_of = [&](int k) {
        return (m.sell_ptr[c0 + k + 1] - m.sell_ptr[c0 + k] + m.sell_bptr[c0 + k + 1] - m.sell_bptr[c0 + k]) >> 5;
    };
    const size_t room = (a.smem - vectors) / pcg_slot_bytes<R>();
    int cap = 0;
    for (int most = 1 << 12; most > 0; most >>= 1) {
        size_t need = 0;
        for (int k = 0; k < nc; ++k) need += min(max(slots_of(k) - KR * sub, 0), cap + most);
        if (need <= room && cap + most <= MS * sub) cap += most;
    }
    int before = 0; // resident slots of the chunks before this one
    for (int k = 0; k < ch && k < nc; ++k) before += min(max(slots_of(k) - KR * sub, 0), cap);
    const int rs0 = KR * sub, rs1 = rs0 + min(max(ns - rs0, 0), cap); // the chunk's slots in shared memory
    R* const sv = reinterpret_cast<R*>(rest) + 288 * static_cast<size_t>(before + part); // the warp's first slot
    const int nsm = rs1 > rs0 + part ? (rs1 - rs0 - part + sub - 1) / sub : 0;         // its slots there
    // Slot q of the chunk, this lane's block (transposed where borrowed) and the index of its column.
    const auto load_slot = [&](int q, R k9[9], int& at) {
        const bool own = q < w0;
        const int2 ref = own ? make_int2(9 * s0 + 288 * q + lane, 0) : __ldg(m.sell_bref + t0 + 32 * (q - w0) + lane);
        at = !(free & 8u) ? 0 : own ? plan.idx_own[s0 + 32 * q + lane]
                                  : plan.idx_bor[t0 + 32 * (q - w0) + lane];
        R v[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) v[e] = __ldg(a.val + static_cast<size_t>(ref.x) + 32 * e);
#pragma unroll
        for (int e = 0; e < 9; ++e) k9[e] = own ? v[e] : v[3 * (e % 3) + e / 3];
    };
    R kr[KR > 0 ? KR : 1][9];
    int ki[KR > 0 ? KR : 1];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        ki[j] = 0;
#pragma unroll
        for (int e = 0; e < 9; ++e) kr[j][e] = R(0);
        if (part + j * sub < ns) load_slot(part + j * sub, kr[j], ki[j]);
    }
    unsigned packed[MS / 2]; // two 16-bit column indices each
#pragma unroll
    for (int j = 0; j < MS; ++j) {
        if ((j & 1) == 0) packed[j / 2] = 0;
        if (j < nsm) {
            R k9[9];
            int at;
            load_slot(rs0 + part + sub * j, k9, at);
            store_block(sv + 288 * static_cast<size_t>(sub * j), lane, k9);
            packed[j / 2] |= static_cast<unsigned>(at) << (16 * (j & 1));
        }
    }
    for (int i = tid; i < L; i += kPcgThreads) list[i] = plan.halo[static_cast<size_t>(plan.halo_stride) * block + i];
    for (int i = tid; i < PS * (own_rows + L); i += kPcgThreads) ps[i] = R(0);
    for (int i = tid; i < 2 * kPcgWarps; i += kPcgThreads) red[i] = 0.0;
    // The row's state.
    const int row = on && part == 0 ? lane_row : -1;
    R x[3] = {0, 0, 0}, r[3] = {0, 0, 0}, z[3] = {0, 0, 0}, p[3] = {0, 0, 0}, D[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) D[t] = R(0);
    if (row >= 0) {
        ld3<4>(a.b4, row, r);
        R mk[3];
        ld3<4>(a.mask4, row, mk);
#pragma unroll
        for (int i = 0; i < 3; ++i) free |= mk[i] != R(0) ? 1u << i : 0u;
        R d[4]; // the symmetric block's upper triangle
        ld4(a.dinv + 12 * static_cast<size_t>(row), d);
        D[0] = d[0], D[1] = d[1], D[2] = d[2];
        ld4(a.dinv + 12 * static_cast<size_t>(row) + 4, d);
        D[3] = d[1], D[4] = d[2];
        ld4(a.dinv + 12 * static_cast<size_t>(row) + 8, d);
        D[5] = d[2];
    }
    unsigned number = __ldcg(a.number + grp);
    if (tid == 0) *s_lost = 0;
    __syncthreads();
    // z = D r, published under the next iteration's number.
    const auto publish_z = [&]() {
        ++number;
        z[0] = D[0] * r[0] + D[1] * r[1] + D[2] * r[2];
        z[1] = D[1] * r[0] + D[3] * r[1] + D[4] * r[2];
        z[2] = D[2] * r[0] + D[4] * r[1] + D[5] * r[2];
        if (row >= 0 && blocks > 1) publish3(a.z4 + 4 * static_cast<size_t>(row), z, number);
    };
    // z of the halo, waiting for each word; G words are in flight per thread.
    const auto each_halo = [&](auto&& use) {
        for (int i0 = tid; i0 < L; i0 += G * kPcgThreads) {
            Pending<R> zv[G];
            unsigned missing = 0;
#pragma unroll
            for (int j = 0; j < G; ++j)
                if (i0 + j * kPcgThreads < L) missing |= 1u << j;
            for (unsigned spin = 0; missing != 0; ++spin) {
                if (spin >= a.polls) {
                    *s_lost = 1;
                    break;
                }
#pragma unroll
                for (int j = 0; j < G; ++j)
                    if ((missing >> j) & 1u) zv[j].load(a.z4 + 4 * static_cast<size_t>(list[i0 + j * kPcgThreads]));
#pragma unroll
                for (int j = 0; j < G; ++j)
                    if (((missing >> j) & 1u) && zv[j].ready(number)) {
                        missing &= ~(1u << j);
                        R t[3];
                        zv[j].get(t);
                        use(i0 + j * kPcgThreads, t);
                    }
            }
        }
    };
    // p = z + beta p of a vertex of the halo, as its owner forms it.
    const auto advance = [&](int i, const R t[3], R be) {
        R* at = ps + PS * static_cast<size_t>(own_rows + i);
        R v[3];
        lds3(at, v);
#pragma unroll
        for (int e = 0; e < 3; ++e) v[e] = fma(be, v[e], t[e]);
        sts3(at, v);
    };
    // The block's sums of NV values, published by warp v as value first + v; then warp v + NV j polls and adds
    // value v of blocks 32 j to 32 j + 31 (one word a lane: five in flight cost the loop 30 registers).
    const auto publish_sums = [&](int nv, int first) {
        if (warp >= nv) return;
        double b = lane < kPcgWarps ? red[kPcgWarps * warp + lane] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) b = shfl_xor_add(b, b, o);
        if (lane != 0) return;
        if (blocks > 1)
            st_word(a.words + static_cast<size_t>(first + warp) * plan.blocks + block, __double2loint(b), __double2hiint(b), 0u,
                    number);
        else
            total[warp] = b;
    };
    const auto poll_sums = [&](int nv, int first) {
        const int val = warp % nv, from = 32 * (warp / nv);
        if (blocks <= 1 || from >= blocks) return;
        double b = 0;
        if (from + lane < blocks) {
            const uint4* at = a.words + static_cast<size_t>(first + val) * plan.blocks + g.b0 + from + lane;
            uint4 u = ld_word(at);
            for (unsigned spin = 0; u.w != number; ++spin) {
                if (spin >= a.polls) {
                    *s_lost = 1;
                    break;
                }
                u = ld_word(at);
            }
            b = __hiloint2double(u.y, u.x);
        }
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = shfl_xor_add(b, b, o);
        if (lane == 0) total[warp] = b;
    };
    static_assert(2 * ((kPcgMaxBlocks + 31) / 32) <= kPcgWarps, "a warp for each value of 32 blocks");
    const auto sum_of = [&](int nv, int v) {
        double t = total[v];
        for (int k = 1; 32 * k < blocks; ++k) t += total[nv * k + v];
        return t;
    };
    int iters = 0, breakdown = 0;
    double rr = 0, gamma = 1;
    bool lost = false;
    publish_z();
    for (;;) {
        // gamma = r.z and r.r: over the warp (lanes 0 and 16 end with one each), the block, the group.
        {
            double v0 = 0, v1 = 0;
            if (row >= 0)
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    v0 += static_cast<double>(r[i]) * z[i];
                    v1 += static_cast<double>(r[i]) * r[i];
                }
            const bool up = lane & 16;
            double t = shfl_xor_add(up ? v1 : v0, up ? v0 : v1, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) t = shfl_xor_add(t, t, o);
            if (part == 0 && (lane & 15) == 0) red[kPcgWarps * (lane >> 4) + warp] = t;
        }
        __syncthreads();
        publish_sums(2, 0);
        if (tid == kPcgThreads - 1) scal[0] = 1.0 / gamma; // off the path between two exchanges
        if (staged)
            each_halo([&](int i, const R t[3]) {
#pragma unroll
                for (int e = 0; e < 3; ++e) parts[3 * static_cast<size_t>(i) + e] = t[e];
            });
        poll_sums(2, 0);
        __syncthreads();
        gamma = sum_of(2, 0), rr = sum_of(2, 1);
        lost = *s_lost != 0;
        if (lost) break;
        if (iters == 0) {
            const double tol = a.tols != nullptr ? a.tols[grp] : a.tol;
            if (tid == 0) scal[1] = tol * tol * rr, scal[2] = rr;
            if (rr == 0.0 || a.max_iters <= 0) break;
        } else if (rr <= scal[1] || iters >= a.max_iters || !isfinite(rr)) {
            break;
        }
        const R be = iters > 0 ? static_cast<R>(gamma * scal[0]) : R(0);
#pragma unroll
        for (int i = 0; i < 3; ++i) p[i] = fma(be, p[i], z[i]);
        if (on && part == 0) sts3(ps + PS * static_cast<size_t>(32 * ch + lane), p);
        if (staged) {
            for (int i = tid; i < L; i += kPcgThreads) advance(i, parts + 3 * static_cast<size_t>(i), be);
        } else {
            each_halo([&](int i, const R t[3]) { advance(i, t, be); });
        }
        __syncthreads();
        R y[3] = {0, 0, 0};
        const auto product = [&](const R k9[9], int at) {
            R v[3];
            lds3(ps + PS * static_cast<size_t>(at), v);
            y[0] += k9[0] * v[0] + k9[1] * v[1] + k9[2] * v[2];
            y[1] += k9[3] * v[0] + k9[4] * v[1] + k9[5] * v[2];
            y[2] += k9[6] * v[0] + k9[7] * v[1] + k9[8] * v[2];
        };
#pragma unroll
        for (int j = 0; j < KR; ++j)
            if (part + j * sub < ns) product(kr[j], ki[j]);
#pragma unroll
        for (int j = 0; j < MS; ++j) {
            if (j >= nsm) break;
            R k9[9];
            load_block(sv + 288 * static_cast<size_t>(sub * j), lane, k9);
            product(k9, static_cast<int>((packed[j / 2] >> (16 * (j & 1))) & 0xffffu));
        }
#pragma unroll 1
        for (int q = rs0 + part + sub * nsm; q < ns; q += sub) {
            R k9[9];
            int at;
            load_slot(q, k9, at);
            product(k9, at);
        }
        if (sub > 1) { // the chunk's parts, added in order by its first warp
            if (part != 0)
#pragma unroll
                for (int i = 0; i < 3; ++i) parts[96 * warp + 32 * i + lane] = y[i];
            __syncthreads();
            if (part == 0)
                for (int k = 1; k < sub; ++k)
#pragma unroll
                    for (int i = 0; i < 3; ++i) y[i] += parts[96 * (warp + k) + 32 * i + lane];
        }
        {
            double v = 0;
            if (row >= 0)
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    y[i] = (free >> i) & 1u ? y[i] : R(0);
                    v += static_cast<double>(p[i]) * y[i];
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = shfl_xor_add(v, v, o);
            if (part == 0 && lane == 0) red[warp] = v;
        }
        __syncthreads();
        publish_sums(1, 2);
        poll_sums(1, 2);
        __syncthreads();
        const double pAp = sum_of(1, 0);
        lost = *s_lost != 0;
        if (lost) break;
        if (!(pAp > 0.0) || !isfinite(pAp)) {
            breakdown = 1;
            if (iters == 0 && a.first_direction)
#pragma unroll
                for (int i = 0; i < 3; ++i) x[i] = p[i];
            break;
        }
        const R al = static_cast<R>(gamma / pAp);
#pragma unroll
        for (int i = 0; i < 3; ++i) r[i] = fma(-al, y[i], r[i]);
        publish_z();
#pragma unroll
        for (int i = 0; i < 3; ++i) x[i] = fma(al, p[i], x[i]); // while the words travel
        ++iters;
    }
    if (row >= 0) st4(a.x4 + 4 * static_cast<size_t>(row), x[0], x[1], x[2]);
    if (rank == 0 && tid == 0) {
        PcgState* st = a.st + grp;
        st->rr = rr;
        st->bb = scal[2];
        st->iters = iters;
        st->breakdown = breakdown;
        st->done = 1;
        a.number[grp] = number;
    }
    if (lost && tid == 0) a.st[grp].lost = 1;
}

} // namespace
} // namespace lpg
