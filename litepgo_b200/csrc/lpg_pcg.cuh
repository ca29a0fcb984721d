// lpg_pcg.cuh -- block-Jacobi PCG of a whole solve in one cooperative launch, for meshes whose rows fit
// one sliced-ELL chunk per warp (16 per block, one block per SM). Included by lpg_solve.cu, whose vector
// helpers and PcgState it uses.
//
// The launch-per-step iteration (spmv_sell and pcg_update in a graph) is bound at these sizes by its two
// launches and its chain of gathers and reductions through L2. Here a lane keeps its row's x, r, p, s and
// preconditioner block in registers for the whole solve, and a block its chunks' matrix values as far as
// they fit (both triangles, borrowed blocks transposed once): the first slots of a warp in registers, up to
// 16 more in shared memory, the rest read from L2. What crosses blocks is z and three sums:
// - z = D r of the block's rows and their neighbours (the halo) is staged in shared memory. A vertex's z is
//   one 16-byte word (two in FP64) that carries the iteration's number, so a reader polls the word itself:
//   no fence, no flag, one L2 round trip.
// - CG in the form with one reduction (Chronopoulos and Gear, below): gamma, delta and r.r of a block are
//   published as numbered words too, and three warps of every block poll all of them and add them in block
//   order, so that all blocks hold bitwise the same sums and results do not depend on scheduling.
// Between the two exchanges every block has read what it waits for, so z is kept once and the sums twice
// (by the number's parity). An iteration is then two L2 round trips, the products and FP64 latency.
//
// Measured per iteration, B200 (launch-per-step, then this kernel): 648 vertices FP64 14.2 and 4.5 us;
// 4,896 FP64 16.4 and 6.4; 62,197 FP32 15.6 and 9.3, where the products (18 slots a lane) and the wait for
// the slowest block are half. A build that spilled 300 bytes a thread took 14 at the last: beside 227 KB of
// shared memory the L1 holds no spills, hence KR, G and the scalars in shared memory below.
#pragma once

namespace lpg {
namespace {

constexpr int kPcgThreads = 512, kPcgWarps = kPcgThreads / 32;
constexpr int kPcgMaxBlocks = 160;     // five slots per polling lane
constexpr unsigned kPcgSpins = 1u << 22; // polls of one exchange before it gives up (seconds)

// Plan of the launch, built once per handle: per block the vertices whose direction it keeps (its
// columns, ascending) and every slot's index into that list (indexed as sell_col and sell_bref).
struct PcgPlan {
    int blocks = 0, halo_stride = 0;
    const int32_t* halo = nullptr;       // [blocks][halo_stride]
    const int32_t* halo_count = nullptr; // [blocks]
    const uint16_t* idx_own = nullptr;
    const uint16_t* idx_bor = nullptr;
};
__host__ __device__ inline int pcg_first_chunk(int n_sell, int blocks, int b) {
    return static_cast<int>(static_cast<int64_t>(n_sell) * b / blocks);
}

// One block per plan block: marks the columns of its chunks in a bitmap over the vertices, numbers them
// in ascending order and writes the list (when halo is not null) and the slots' indices.
__global__ void __launch_bounds__(kPcgThreads) pcg_plan_kernel(const DevMesh m, int blocks, int32_t* halo, int stride,
                                                               int32_t* count, uint16_t* idx_own, uint16_t* idx_bor) {
    extern __shared__ unsigned s_bits[]; // bitmap, then the number of marks before each word
    const int words = (m.V + 31) / 32;
    unsigned* before = s_bits + words;
    __shared__ unsigned s_sum[kPcgWarps];
    __shared__ unsigned s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < words; i += kPcgThreads) s_bits[i] = 0;
    if (tid == 0) s_base = 0;
    __syncthreads();
    const int c0 = pcg_first_chunk(m.n_sell, blocks, blockIdx.x), c1 = pcg_first_chunk(m.n_sell, blocks, blockIdx.x + 1);
    const int o0 = m.sell_ptr[c0], o1 = m.sell_ptr[c1], b0 = m.sell_bptr[c0], b1 = m.sell_bptr[c1];
    for (int c = c0 + warp; c < c1; c += kPcgWarps) {
        const int row = m.sell_row[32 * static_cast<size_t>(c) + lane];
        if (row >= 0) atomicOr(s_bits + (row >> 5), 1u << (row & 31));
    }
    for (int i = o0 + tid; i < o1; i += kPcgThreads) atomicOr(s_bits + (m.sell_col[i] >> 5), 1u << (m.sell_col[i] & 31));
    for (int i = b0 + tid; i < b1; i += kPcgThreads) atomicOr(s_bits + (m.sell_bref[i].y >> 5), 1u << (m.sell_bref[i].y & 31));
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
        for (; b; b &= b - 1) halo[static_cast<size_t>(stride) * blockIdx.x + at++] = 32 * i + __ffs(b) - 1;
    }
    auto rank = [&](int v) {
        return static_cast<uint16_t>(before[v >> 5] + __popc(s_bits[v >> 5] & ((1u << (v & 31)) - 1u)));
    };
    for (int i = o0 + tid; i < o1; i += kPcgThreads) idx_own[i] = rank(m.sell_col[i]);
    for (int i = b0 + tid; i < b1; i += kPcgThreads) idx_bor[i] = rank(m.sell_bref[i].y);
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

// Values per staged vertex: float4 in FP32, three doubles in FP64.
template <typename R> constexpr int pcg_stride() { return sizeof(R) == 4 ? 4 : 3; }
// Shared memory of the staged z and its vertex list.
template <typename R> constexpr size_t pcg_halo_bytes(int n) {
    return (static_cast<size_t>(n) * (pcg_stride<R>() * sizeof(R) + sizeof(int32_t)) + 15) / 16 * 16;
}
// Shared memory of one slot of a chunk (32 blocks).
template <typename R> constexpr size_t pcg_slot_bytes() { return 32 * 9 * sizeof(R); }
constexpr size_t kPcgFixed = (4 * kPcgWarps + 16 + 3 * 32 * kPcgWarps) * sizeof(double); // sums, split rows' parts

template <typename R> struct PcgArgs {
    const R *val, *dinv, *mask4, *b4;
    R *x4, *z4;
    PcgState* st;
    uint4* words;     // [2][3][blocks]
    unsigned* number; // exchanges so far (device)
    double tol;
    int max_iters;
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

// The iteration is CG with one reduction (Chronopoulos and Gear, "s-step iterative methods for symmetric
// linear systems", 1989): with w = A z, gamma = r.z and delta = z.w, p^T A p = delta - beta gamma / alpha_old,
// and A p follows from A z by the recurrence of p itself, s = w + beta s.
template <typename R>
__global__ void __launch_bounds__(kPcgThreads, 1) pcg_solve_kernel(const DevMesh m, const PcgPlan plan, const PcgArgs<R> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int PS = pcg_stride<R>(), KR = sizeof(R) == 4 ? 2 : 0, G = sizeof(R) == 4 ? 2 : 1;
    constexpr int MS = 16; // most slots of a warp in shared memory (their column indices are in registers)
    double* red = reinterpret_cast<double*>(smem_raw); // [4 values][warps], then the three sums
    double* total = red + 4 * kPcgWarps;
    volatile int* s_lost = reinterpret_cast<volatile int*>(total + 4);
    // Scalars of thread 0: 1 / gamma and 1 / alpha of the iteration before (by parity), then its gamma and
    // p.Ap, the squared tolerance and |b|^2.
    double* scal = total + 8;
    R* parts = reinterpret_cast<R*>(total + 16); // [warp][3][32]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int blocks = plan.blocks;
    const int c0 = pcg_first_chunk(m.n_sell, blocks, blockIdx.x), c1 = pcg_first_chunk(m.n_sell, blocks, blockIdx.x + 1);
    const int nc = c1 - c0; // at most kPcgWarps
    const int L = plan.halo_count[blockIdx.x];
    R* zs = reinterpret_cast<R*>(smem_raw + kPcgFixed);
    int32_t* list = reinterpret_cast<int32_t*>(zs + static_cast<size_t>(PS) * L);
    unsigned char* rest = smem_raw + kPcgFixed + pcg_halo_bytes<R>(L);
    // `sub` warps share a chunk (its slots dealt round robin); the first of them owns the rows.
    int sub = 1;
    while (2 * sub * nc <= kPcgWarps && sub < 4) sub *= 2;
    const int ch = warp / sub, part = warp - sub * ch;
    const bool on = ch < nc;
    const int c = c0 + (on ? ch : 0);
    const int s0 = m.sell_ptr[c], w0 = (m.sell_ptr[c + 1] - s0) >> 5;
    const int t0 = m.sell_bptr[c], bw = (m.sell_bptr[c + 1] - t0) >> 5;
    const int ns = on ? w0 + bw : 0;
    // Of a chunk's slots (own, then borrowed) the first KR of each of its warps are in registers, as many
    // more as fit are in shared memory (at most `cap` per chunk, the largest cap that fits all chunks: the
    // same walk in every thread), the rest are read from L2.
    const auto slots_of = [&](int k) {
        return (m.sell_ptr[c0 + k + 1] - m.sell_ptr[c0 + k] + m.sell_bptr[c0 + k + 1] - m.sell_bptr[c0 + k]) >> 5;
    };
    const size_t room = (a.smem - kPcgFixed - pcg_halo_bytes<R>(L)) / pcg_slot_bytes<R>();
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
        at = own ? plan.idx_own[s0 + 32 * q + lane] : plan.idx_bor[t0 + 32 * (q - w0) + lane];
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
    for (int i = tid; i < L; i += kPcgThreads) list[i] = plan.halo[static_cast<size_t>(plan.halo_stride) * blockIdx.x + i];
    for (int i = tid; i < 4 * kPcgWarps; i += kPcgThreads) red[i] = 0.0;
    // The row's state.
    const int row = on && part == 0 ? m.sell_row[32 * static_cast<size_t>(c) + lane] : -1;
    R x[3] = {0, 0, 0}, r[3] = {0, 0, 0}, z[3] = {0, 0, 0}, p[3] = {0, 0, 0}, s[3] = {0, 0, 0}, D[6];
    unsigned free = 0; // bit i: component i of the row is free
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
    unsigned number = __ldcg(a.number);
    if (tid == 0) *s_lost = 0;
    if (blockIdx.x == 0 && tid == 0) a.st->lost = 0;
    __syncthreads();
    int iters = 0, breakdown = 0;
    bool lost = false;
    for (;;) {
        // z = D r, published under this iteration's number.
        ++number;
        z[0] = D[0] * r[0] + D[1] * r[1] + D[2] * r[2];
        z[1] = D[1] * r[0] + D[3] * r[1] + D[4] * r[2];
        z[2] = D[2] * r[0] + D[4] * r[1] + D[5] * r[2];
        if (row >= 0) publish3(a.z4 + 4 * static_cast<size_t>(row), z, number);
        if (tid == 0) { // off the path between two exchanges: 1 / gamma and 1 / alpha = p.Ap / gamma
            double* next = scal + 2 * (iters & 1);
            const double ig = iters > 0 ? 1.0 / scal[4] : 0.0;
            next[0] = ig;
            next[1] = iters > 0 ? scal[5] * ig : 0.0;
        }
        // z of the block's rows and their neighbours, waiting for each word; G words are in flight per thread.
        for (int i0 = tid; i0 < L; i0 += G * kPcgThreads) {
            Pending<R> zv[G];
            unsigned missing = 0;
#pragma unroll
            for (int j = 0; j < G; ++j)
                if (i0 + j * kPcgThreads < L) missing |= 1u << j;
            for (unsigned spin = 0; missing != 0; ++spin) {
                if (spin >= kPcgSpins) {
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
                        sts3(zs + PS * static_cast<size_t>(i0 + j * kPcgThreads), t);
                    }
            }
        }
        __syncthreads();
        R y[3] = {0, 0, 0};
        const auto product = [&](const R k9[9], int at) {
            R v[3];
            lds3(zs + PS * static_cast<size_t>(at), v);
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
        // The sums gamma = r.z, delta = z.w and r.r over the block: a transposed tree over the warp (lane
        // group lane / 8 ends with value lane / 8), then over the warps.
        double gamma, delta;
        {
            double v[3] = {0, 0, 0};
            if (row >= 0)
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    y[i] = (free >> i) & 1u ? y[i] : R(0);
                    v[0] += static_cast<double>(r[i]) * z[i];
                    v[1] += static_cast<double>(z[i]) * y[i];
                    v[2] += static_cast<double>(r[i]) * r[i];
                }
            const bool up = lane & 16, mid = lane & 8;
            const double k0 = shfl_xor_add(up ? v[2] : v[0], up ? v[0] : v[2], 16);
            const double k1 = shfl_xor_add(up ? 0.0 : v[1], up ? v[1] : 0.0, 16);
            double t = shfl_xor_add(mid ? k1 : k0, mid ? k0 : k1, 8);
            t = shfl_xor_add(t, t, 4);
            t = shfl_xor_add(t, t, 2);
            t = shfl_xor_add(t, t, 1);
            if (part == 0 && (lane & 7) == 0) red[kPcgWarps * (lane >> 3) + warp] = t;
            __syncthreads();
            uint4* all = a.words + static_cast<size_t>(number & 1u) * 3 * blocks;
            if (warp < 3) { // warp v: the block's value v, then everyone's
                static_assert(kPcgWarps == 16, "one value per lane below 16");
                double b = lane < kPcgWarps ? red[kPcgWarps * warp + lane] : 0.0;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) b = shfl_xor_add(b, b, o);
                if (lane == 0) st_word(all + blocks * warp + blockIdx.x, __double2loint(b), __double2hiint(b), 0u, number);
                constexpr int kPer = kPcgMaxBlocks / 32;
                double g[kPer];
                unsigned missing = 0;
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    g[j] = 0;
                    if (lane + 32 * j < blocks) missing |= 1u << j;
                }
                for (unsigned spin = 0; missing != 0; ++spin) {
                    if (spin >= kPcgSpins) {
                        *s_lost = 1;
                        break;
                    }
                    uint4 u[kPer];
#pragma unroll
                    for (int j = 0; j < kPer; ++j)
                        if ((missing >> j) & 1u) u[j] = ld_word(all + blocks * warp + lane + 32 * j);
#pragma unroll
                    for (int j = 0; j < kPer; ++j)
                        if (((missing >> j) & 1u) && u[j].w == number) {
                            g[j] = __hiloint2double(u[j].y, u[j].x);
                            missing &= ~(1u << j);
                        }
                }
                __syncwarp();
                double sum = 0;
#pragma unroll
                for (int j = 0; j < kPer; ++j) sum += g[j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum = shfl_xor_add(sum, sum, o);
                if (lane == 0) total[warp] = sum;
            }
            __syncthreads();
            gamma = total[0], delta = total[1];
            lost = *s_lost != 0;
        }
        if (lost) break;
        {
            const double rr = total[2];
            if (iters == 0) {
                if (tid == 0) scal[6] = a.tol * a.tol * rr, scal[7] = rr;
                if (rr == 0.0 || a.max_iters <= 0) break;
            } else if (rr <= scal[6] || iters >= a.max_iters || !isfinite(rr)) {
                break;
            }
        }
        const double beta = gamma * scal[2 * (iters & 1)];
        const double pAp = fma(-beta * gamma, scal[2 * (iters & 1) + 1], delta);
        if (!(pAp > 0.0) || !isfinite(pAp)) {
            breakdown = 1;
            // Negative curvature on the first step: the preconditioned residual is the direction.
            if (iters == 0)
#pragma unroll
                for (int i = 0; i < 3; ++i) x[i] = z[i];
            break;
        }
        const double alpha = gamma / pAp;
        const R al = static_cast<R>(alpha), be = static_cast<R>(beta);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            p[i] = z[i] + be * p[i];
            s[i] = y[i] + be * s[i];
            x[i] += al * p[i];
            r[i] = r[i] - al * s[i];
        }
        ++iters;
        if (tid == 0) scal[4] = gamma, scal[5] = pAp;
    }
    if (row >= 0) st4(a.x4 + 4 * static_cast<size_t>(row), x[0], x[1], x[2]);
    if (blockIdx.x == 0 && tid == 0) {
        a.st->rr = total[2];
        a.st->bb = scal[7];
        a.st->iters = iters;
        a.st->breakdown = breakdown;
        a.st->done = 1;
        *a.number = number;
    }
    if (lost && tid == 0) a.st->lost = 1;
}

} // namespace
} // namespace lpg
