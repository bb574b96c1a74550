// Uneven batches: products of different ring sizes and moduli in one graph.
//
// pm_batch_create builds, once, everything a run needs: a plan per product
// (prime basis sized for its N and bits(q), CRT constants and weights),
// packed device buffers for a, b, c and the residue planes, per-product tensor
// maps, and flat work tables:
//   conversion items  (product, polynomial, column group) per number of folded
//                     column stages (three, two or one, by the product's basis) --
//                     one persistent launch of k1f_convert per class, each on its
//                     share of the SMs; in batches of few tiles (product, prime
//                     group, polynomial, column group) ordered prime group first --
//                     one persistent launch of k1t_convert;
//   row items         (product, prime, first row) per ring size class -- one
//                     launch per class: the persistent k2p_rows for rows of
//                     1024 values or more (items prime/row first, so a CTA
//                     stages a row's twiddles once for every product that
//                     has it), k2w_rows for shorter rows;
//   CRT items         (product, column group) per width class -- one persistent
//                     launch of k3t_crt per class.
// These launches are captured into a CUDA graph (the classes of a phase on
// parallel branches), so pm_batch_run is a single cudaGraphLaunch.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <vector>

#include "../../include/polymul.h"
#include "pm_internal.h"
#include "rows_persistent.cuh"
#include "rows_warp.cuh"
#include "convert_fold.cuh"
#include "tensor_kernels.cuh"

namespace pm {

// conversion tiles of one class from a table of (product, polynomial, column group) items
struct TableFoldWork {
    const uint4* items;
    int nitems;
    const BatchProduct* prod;
    const CUtensorMap* maps;  // [3 * products]: a, b, residues
    uint32_t* work;
    PlainRows plain;  // (not used: batches have 16-byte coefficient rows)
    __device__ int total() const { return nitems; }
    __device__ TileItem item(int k) const {
        const uint4 v = items[k];
        return TileItem{int(v.x), int(v.y), int(v.z)};
    }
    __device__ ConvTarget target(int z, int poly) const {
        const BatchProduct& d = prod[z];
        return ConvTarget{maps + 3 * z + poly, 0, work + d.ws_off, d.n, d.logC, d.P};
    }
};

// the same work by K1T: (product, prime group, polynomial, column group) items of every class
struct TableConvWork {
    const uint4* items;
    int nitems;
    const BatchProduct* prod;
    const CUtensorMap* maps;
    uint32_t* work;
    __device__ int total() const { return nitems; }
    __device__ ConvItem item(int k) const {
        const uint4 v = items[k];
        return ConvItem{int(v.x), int(v.y), int(v.z), int(v.w)};
    }
    __device__ ConvTarget target(int z, int poly) const {
        const BatchProduct& d = prod[z];
        return ConvTarget{maps + 3 * z + poly, 0, work + d.ws_off, d.n, d.logC, d.P};
    }
    __device__ int2 range(int b, int grid) const {  // contiguous runs of the table
        const int chunk = (nitems + grid - 1) / grid;
        return make_int2(min(nitems, b * chunk), min(nitems, (b + 1) * chunk));
    }
};

// Tiles of 128 coefficients an SM up to which a batch converts by K1T.  K1F's CTAs fill an SM and load
// 128 KB of weights each before their first tile, a launch per class; K1T is one launch of small CTAs,
// three an SM, that share a tile's primes out.  Whole batches, K1T / K1F: one product of 256, 868 bits,
// 16.4 / 22.6 us; eight of 1024 (128 tiles) 20.6 / 24.6; four of 192 .. 590 bits (312) 27.8 / 33.2;
// two of 8192 (256) 28.7 / 28.7.  Past the line either: four of 8192, 400 bits (512), 28.7 / 26.7;
// eight of 4096, 600 bits (512), 30.8 / 32.8; 64 of 1024 (1024) 55.4 / 53.3.
constexpr int kBatchTilesPerSm = 3;

// rows of one size class from a table of (product, prime, first row) items
struct TableRowWork {
    const uint4* items;
    int nitems;
    const BatchProduct* prod;
    uint32_t* work;
    __device__ int total() const { return nitems; }
    __device__ RowItem item(int k) const {
        const uint4 v = items[k];
        const BatchProduct& d = prod[v.x];
        return RowItem{int(v.y), int(v.z), work + d.ws_off + size_t(v.y) * d.n + (size_t(v.z) << d.logC),
                       size_t(d.P) * d.n};
    }
};

namespace {

int sm_count_dev() {
    int dev = 0, count = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    return count ? count : 148;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        cuda_check(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q),
                   "look up cuTensorMapEncodeTiled");
        if (!p || q != cudaDriverEntryPointSuccess) throw Failure(PM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

CUtensorMap encode(CUtensorMapDataType type, const void* base, const cuuint64_t dims[4], const cuuint64_t strides[3],
                   const cuuint32_t box[4], CUtensorMapSwizzle swizzle) {
    CUtensorMap map;
    const cuuint32_t es[4] = {1, 1, 1, 1};
    const CUresult r = encode_tiled()(&map, type, 4, const_cast<void*>(base), dims, strides, box, es,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Failure(PM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a batch product");
    return map;
}

template <int LOGF>
void launch_fold_class(const TableFoldWork& w, int ctas, int qbytes, const DeviceBasis& B, uint32_t* err,
                       cudaStream_t st) {
    cuda_check(cudaFuncSetAttribute(k1f_convert<LOGF, TableFoldWork>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(k1f_smem_bytes())),
               "batch conversion shared memory");
    k1f_convert<LOGF, TableFoldWork><<<ctas, k1f_threads(false), k1f_smem_bytes(), st>>>(
        w, B.d_pc, B.d_fold_weights + (LOGF - 1) * size_t(kFoldWeightBytes), B.d_tw_fwd, qbytes, err);
}

template <int LOGC, int KP>
void launch_rows_class(const uint4* items, int count, const BatchProduct* prod, uint32_t* work, const DeviceBasis& B,
                       uint32_t* err, cudaStream_t st) {
    const TableRowWork w{items, count, prod, work};
    if constexpr (LOGC >= 10) {
        const size_t smem = k2p_smem_bytes(LOGC);
        cuda_check(cudaFuncSetAttribute(k2p_rows<LOGC, KP, TableRowWork>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(smem)),
                   "batch row shared memory");
        const int ctas = std::min(count, sm_count_dev() * k2p_min_blocks(LOGC));
        k2p_rows<LOGC, KP, TableRowWork><<<ctas, k2p_threads(LOGC, KP), smem, st>>>(w, B.d_pc, B.d_tw_fwd,
                                                                                    B.d_tw_inv, 4, err);
    } else {
        k2w_rows<LOGC, TableRowWork><<<k2w_grid(count, sm_count_dev()), 32 * kWarpRowWarps, k2w_smem_bytes<LOGC>(),
                                       st>>>(w, B.d_pc, B.d_tw_fwd, B.d_tw_inv, 4);
    }
}

// radix_log: the register-pass radix of the persistent kernel's rows (C >= 1024)
template <int LOGC>
void launch_rows_radix(int radix_log, const uint4* items, int count, const BatchProduct* prod, uint32_t* work,
                       const DeviceBasis& B, uint32_t* err, cudaStream_t st) {
    if constexpr (LOGC < 10)
        launch_rows_class<LOGC, 4>(items, count, prod, work, B, err, st);
    else if (radix_log == 2)
        launch_rows_class<LOGC, 2>(items, count, prod, work, B, err, st);
    else if (radix_log == 3)
        launch_rows_class<LOGC, 3>(items, count, prod, work, B, err, st);
    else
        launch_rows_class<LOGC, 4>(items, count, prod, work, B, err, st);
}

void launch_rows_any(int logC, int radix_log, const uint4* items, int count, const BatchProduct* prod,
                     uint32_t* work, const DeviceBasis& B, uint32_t* err, cudaStream_t st) {
    switch (logC) {
        case 4: return launch_rows_radix<4>(radix_log, items, count, prod, work, B, err, st);
        case 5: return launch_rows_radix<5>(radix_log, items, count, prod, work, B, err, st);
        case 6: return launch_rows_radix<6>(radix_log, items, count, prod, work, B, err, st);
        case 7: return launch_rows_radix<7>(radix_log, items, count, prod, work, B, err, st);
        case 8: return launch_rows_radix<8>(radix_log, items, count, prod, work, B, err, st);
        case 9: return launch_rows_radix<9>(radix_log, items, count, prod, work, B, err, st);
        case 10: return launch_rows_radix<10>(radix_log, items, count, prod, work, B, err, st);
        case 11: return launch_rows_radix<11>(radix_log, items, count, prod, work, B, err, st);
        case 12: return launch_rows_radix<12>(radix_log, items, count, prod, work, B, err, st);
        default: throw Failure(PM_ERR_UNSUPPORTED, "row size outside the batch kernels");
    }
}

template <int W>
void launch_crt_class(const TableCrtWork& w, int ctas, const DeviceBasis& B, uint32_t* err, cudaStream_t st) {
    const size_t smem = k3t_smem_bytes<4>(W);
    cuda_check(cudaFuncSetAttribute(k3t_crt<4, W, TableCrtWork>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(smem)),
               "batch CRT shared memory");
    k3t_crt<4, W, TableCrtWork><<<ctas, tc::kCrtThreads, smem, st>>>(w, B.d_pc, B.d_tw_inv, err);
}

void launch_crt_any(int W, const TableCrtWork& w, int ctas, const DeviceBasis& B, uint32_t* err, cudaStream_t st) {
    switch (W) {
        case 4: return launch_crt_class<4>(w, ctas, B, err, st);
        case 8: return launch_crt_class<8>(w, ctas, B, err, st);
        case 12: return launch_crt_class<12>(w, ctas, B, err, st);
        case 16: return launch_crt_class<16>(w, ctas, B, err, st);
        case 20: return launch_crt_class<20>(w, ctas, B, err, st);
        case 24: return launch_crt_class<24>(w, ctas, B, err, st);
        case 28: return launch_crt_class<28>(w, ctas, B, err, st);
        default: throw Failure(PM_ERR_UNSUPPORTED, "unsupported width");
    }
}

}  // namespace

struct BatchCore {
    int device = 0;
    uint32_t count = 0, coef_limbs = 0;
    std::vector<std::unique_ptr<PlanCore>> plans;
    std::vector<uint64_t> io_off;  // u64 words per product
    size_t io_words = 0;           // u64 words of one of a, b, c
    uint64_t* d_a = nullptr;
    uint64_t* d_b = nullptr;
    uint64_t* d_c = nullptr;
    uint32_t* d_work = nullptr;
    BatchProduct* d_prod = nullptr;
    CUtensorMap* d_maps = nullptr;
    uint4* d_conv_items = nullptr;
    uint4* d_row_items = nullptr;
    uint2* d_crt_items = nullptr;
    uint32_t* d_err = nullptr;
    int conv_items = 0;  // of K1T, or none
    struct FoldClass {
        int f, count, ctas, qbytes;
        size_t offset;  // into d_conv_items
    };
    std::vector<FoldClass> fold_classes;
    struct RowClass {
        int logC, radix_log, count;
        size_t offset;  // into d_row_items
    };
    struct CrtClass {
        int W, count;
        size_t offset;  // into d_crt_items
    };
    std::vector<RowClass> row_classes;
    std::vector<CrtClass> crt_classes;
    cudaGraphExec_t graph = nullptr;
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> events;
    int conv_ctas_per_sm = 3;  // persistent grid size of K1T (autotuned)
    int crt_ctas_per_sm = 0;   // of the CRT (0: as many as fit; autotuned)

    ~BatchCore() {
        cudaSetDevice(device);
        if (graph) cudaGraphExecDestroy(graph);
        for (auto s : streams) cudaStreamDestroy(s);
        for (auto e : events) cudaEventDestroy(e);
        cudaFree(d_a);
        cudaFree(d_b);
        cudaFree(d_c);
        cudaFree(d_work);
        cudaFree(d_prod);
        cudaFree(d_maps);
        cudaFree(d_conv_items);
        cudaFree(d_row_items);
        cudaFree(d_crt_items);
        cudaFree(d_err);
    }

    // Issue the three phases on streams[0], classes of a phase on forked streams.
    void enqueue(cudaStream_t st0) {
        const DeviceBasis& B = *plans[0]->basis;
        const int sms = sm_count_dev();
        auto fork = [&](size_t k) {
            cudaStream_t s = streams[1 + k % (streams.size() - 1)];
            cuda_check(cudaEventRecord(events[0], st0), "batch fork");
            cuda_check(cudaStreamWaitEvent(s, events[0], 0), "batch fork");
            return s;
        };
        auto join = [&](cudaStream_t s, size_t k) {
            cudaEvent_t e = events[1 + k % (events.size() - 1)];
            cuda_check(cudaEventRecord(e, s), "batch join");
            cuda_check(cudaStreamWaitEvent(st0, e, 0), "batch join");
        };
        std::vector<cudaStream_t> used;
        if (conv_items) {
            cuda_check(cudaFuncSetAttribute(k1t_convert<4, TableConvWork>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            int(k1t_smem_bytes())),
                       "batch conversion shared memory");
            const TableConvWork w{d_conv_items, conv_items, d_prod, d_maps, d_work};
            k1t_convert<4, TableConvWork><<<std::min(conv_items, sms * conv_ctas_per_sm), tc::kConvThreads,
                                            k1t_smem_bytes(), st0>>>(w, B.d_pc, B.d_conv_weights, B.d_tw_fwd, d_err);
        }
        for (size_t k = 0; k < fold_classes.size(); ++k) {
            const FoldClass& fc = fold_classes[k];
            cudaStream_t s = fork(k);
            const TableFoldWork w{d_conv_items + fc.offset, fc.count, d_prod, d_maps, d_work, PlainRows{}};
            switch (fc.f) {
                case 1: launch_fold_class<1>(w, fc.ctas, fc.qbytes, B, d_err, s); break;
                case 2: launch_fold_class<2>(w, fc.ctas, fc.qbytes, B, d_err, s); break;
                default: launch_fold_class<3>(w, fc.ctas, fc.qbytes, B, d_err, s); break;
            }
            used.push_back(s);
        }
        cuda_check(cudaGetLastError(), "batch conversion launch");
        for (size_t k = 0; k < used.size(); ++k) join(used[k], k);
        used.clear();
        for (size_t k = 0; k < row_classes.size(); ++k) {
            const RowClass& rc = row_classes[k];
            cudaStream_t s = fork(k);
            launch_rows_any(rc.logC, rc.radix_log, d_row_items + rc.offset, rc.count, d_prod, d_work, B, d_err,
                            s);
            used.push_back(s);
        }
        for (size_t k = 0; k < used.size(); ++k) join(used[k], k);
        used.clear();
        for (size_t k = 0; k < crt_classes.size(); ++k) {
            const CrtClass& cc = crt_classes[k];
            cudaStream_t s = fork(k);
            TableCrtWork w{d_crt_items + cc.offset, cc.count, d_prod, d_maps, d_work, reinterpret_cast<uint32_t*>(d_c)};
            launch_crt_any(cc.W, w, std::min(cc.count, sms * k3t_ctas_per_sm(cc.W, crt_ctas_per_sm)), B, d_err, s);
            used.push_back(s);
        }
        for (size_t k = 0; k < used.size(); ++k) join(used[k], k);
        cuda_check(cudaGetLastError(), "batch launches");
    }

    void build(uint32_t cnt, const uint32_t* ns, const uint64_t* const* qs, const uint32_t* q_limbs, uint32_t limbs) {
        count = cnt;
        coef_limbs = limbs;
        if (limbs % 2) throw Failure(PM_ERR_UNSUPPORTED, "batches need an even coef_limbs (16-byte coefficient rows)");
        cuda_check(cudaGetDevice(&device), "cudaGetDevice");
        std::vector<BatchProduct> prod(cnt);
        std::vector<size_t> ws_off(cnt);
        size_t io = 0, ws = 0;
        for (uint32_t z = 0; z < cnt; ++z) {
            if (ns[z] < 256) throw Failure(PM_ERR_UNSUPPORTED, "batched products need n >= 256");
            auto p = std::make_unique<PlanCore>();
            p->init_tables_only(ns[z], qs[z], q_limbs[z], limbs, PM_CONVERT_TENSOR);
            if (p->logR != 4) throw Failure(PM_ERR_UNSUPPORTED, "batched products need 16-row views");
            io_off.push_back(io);
            ws_off[z] = ws;
            io += size_t(p->n) * limbs;
            ws += p->workspace_bytes / 4;
            BatchProduct& d = prod[z];
            d.n = int(p->n);
            d.logC = int(p->logC);
            d.P = int(p->P);
            d.W = int(p->W);
            d.sbits = int(p->qbits);
            d.delta = p->delta;
            d.stride = int(p->stride);
            d.mu_q = p->mu_q;
            d.io_off = 2 * io_off[z];
            d.ws_off = ws_off[z];
            d.scale = p->d_scale;
            d.consts = p->d_consts;
            d.ktab = p->d_ktab;
            d.crt_w = p->d_crt_weights;
            d.kfrac = p->d_kfrac;
            plans.push_back(std::move(p));
        }
        io_words = io;
        cuda_check(cudaMalloc(&d_a, io * 8), "batch a");
        cuda_check(cudaMalloc(&d_b, io * 8), "batch b");
        cuda_check(cudaMalloc(&d_c, io * 8), "batch c");
        cuda_check(cudaMalloc(&d_work, ws * 4), "batch workspace");
        cuda_check(cudaMalloc(&d_err, 4), "batch error word");
        cuda_check(cudaMemset(d_err, 0, 4), "batch error word");
        const int sms = sm_count_dev();
        size_t tiles128 = 0;
        for (auto& p : plans) tiles128 += 2 * size_t(p->n) / tc::kTileM;
        const bool fold = tiles128 > size_t(sms) * kBatchTilesPerSm;  // K1F, or K1T
        // tensor maps: a, b coefficient bytes and residue planes of each product
        std::vector<CUtensorMap> maps(3 * size_t(cnt));
        for (uint32_t z = 0; z < cnt; ++z) {
            const PlanCore& p = *plans[z];
            const cuuint64_t C = 1ull << p.logC, R = 1ull << p.logR, sb = p.stride * 4ull;
            const cuuint32_t Gc = cuuint32_t(C < 8 ? C : 8);
            const int f = fold ? fold_stages(int(p.P), int(p.logC)) : 0;  // K1F: at least one, as n >= 256
            const cuuint64_t cdims[4] = {sb, C, R, 1};
            const cuuint64_t cstr[3] = {sb, sb * C, sb * C * R};
            const cuuint32_t cbox[4] = {fold ? 256u >> f : 128u, 8u << f, 16u >> f, 1};
            const CUtensorMapSwizzle swizzle =
                f <= 1 ? CU_TENSOR_MAP_SWIZZLE_128B : (f == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
            maps[3 * z] = encode(CU_TENSOR_MAP_DATA_TYPE_UINT8, d_a + io_off[z], cdims, cstr, cbox, swizzle);
            maps[3 * z + 1] = encode(CU_TENSOR_MAP_DATA_TYPE_UINT8, d_b + io_off[z], cdims, cstr, cbox, swizzle);
            // box lands as [row][32 or 64 primes][column]: a constant row stride (primes past P read as zero)
            const cuuint64_t rdims[4] = {C, p.P, R, 1};
            const cuuint64_t rstr[3] = {C * R * 4, C * 4, p.workspace_bytes};
            const cuuint32_t rbox[4] = {Gc, cuuint32_t(crt_cap(int(p.W))), cuuint32_t(R), 1};
            maps[3 * z + 2] = encode(CU_TENSOR_MAP_DATA_TYPE_UINT32, d_work + ws_off[z], rdims, rstr, rbox,
                                     CU_TENSOR_MAP_SWIZZLE_NONE);
        }
        // work tables
        std::vector<uint4> conv;
        for (int pg = 0; pg < 4 && !fold; ++pg)
            for (uint32_t z = 0; z < cnt; ++z) {
                const PlanCore& p = *plans[z];
                if (pg * 16 >= int(p.P)) continue;
                for (uint32_t poly = 0; poly < 2; ++poly)
                    for (uint32_t cg = 0; cg < (1u << p.logC) / 8; ++cg) conv.push_back(make_uint4(z, pg, poly, cg));
            }
        conv_items = int(conv.size());
        std::map<int, std::vector<uint4>> conv_by_f;
        std::map<int, int> qbytes_by_f;
        size_t tiles = 0;
        for (uint32_t z = 0; z < cnt && fold; ++z) {
            const PlanCore& p = *plans[z];
            const int f = fold_stages(int(p.P), int(p.logC));
            const uint32_t groups = (1u << p.logC) / (8u << f);
            for (uint32_t poly = 0; poly < 2; ++poly)
                for (uint32_t cg = 0; cg < groups; ++cg) conv_by_f[f].push_back(make_uint4(z, poly, cg, 0));
            qbytes_by_f[f] = std::max(qbytes_by_f[f], int((p.qbits + 7) / 8));
            tiles += 2 * size_t(groups);
        }
        // a CTA fills an SM: the classes run side by side on shares of them by their tiles; the
        // largest takes what the others leave, so that no CTA waits for a second round
        int left = sms;
        size_t largest = 0;
        for (auto& [f, items] : conv_by_f) {
            const int ctas = std::min(int(items.size()), std::max(1, int(size_t(sms) * items.size() / tiles)));
            fold_classes.push_back(FoldClass{f, int(items.size()), ctas, qbytes_by_f[f], conv.size()});
            conv.insert(conv.end(), items.begin(), items.end());
            left -= ctas;
            if (items.size() > size_t(fold_classes[largest].count)) largest = fold_classes.size() - 1;
        }
        if (fold) {
            FoldClass& fc = fold_classes[largest];
            fc.ctas = std::min(fc.count, fc.ctas + left);
        }
        std::map<int, std::vector<uint4>> rows_by_c;
        for (uint32_t z = 0; z < cnt; ++z) {
            const PlanCore& p = *plans[z];
            const int R = 1 << p.logR, rows = p.logC >= 10 ? 1 : warp_rows(int(p.logC), int(p.logR));
            for (uint32_t i = 0; i < p.P; ++i)
                for (int r = 0; r < R; r += rows) rows_by_c[int(p.logC)].push_back(make_uint4(z, i, uint32_t(r), 0));
        }
        std::vector<uint4> row_items;
        for (auto& [logC, items] : rows_by_c) {
            // consecutive items share their (prime, rows): the row kernels keep their twiddles
            std::stable_sort(items.begin(), items.end(), [](const uint4& x, const uint4& y) {
                return x.y != y.y ? x.y < y.y : x.z < y.z;
            });
            // the radix the autotuner picked for plans of this row size; by default radix 16
            // (rows of C >= 1024; shorter rows' passes are fixed)
            int radix_log = 4;
            for (auto& p : plans)
                if (int(p->logC) == logC && p->tune.tuned) radix_log = p->tune.row_radix_log;
            row_classes.push_back(RowClass{logC, radix_log, int(items.size()), row_items.size()});
            row_items.insert(row_items.end(), items.begin(), items.end());
        }
        std::map<int, std::vector<uint2>> crt_by_w;
        for (uint32_t z = 0; z < cnt; ++z) {
            const PlanCore& p = *plans[z];
            for (uint32_t cg = 0; cg < (1u << p.logC) / 8; ++cg) crt_by_w[int(p.W)].push_back(make_uint2(z, cg));
        }
        std::vector<uint2> crt_items;
        for (auto& [W, items] : crt_by_w) {
            crt_classes.push_back(CrtClass{W, int(items.size()), crt_items.size()});
            crt_items.insert(crt_items.end(), items.begin(), items.end());
        }
        auto upload = [](auto** dst, const auto& v, const char* what) {
            using T = std::remove_pointer_t<std::remove_reference_t<decltype(*dst)>>;
            cuda_check(cudaMalloc(dst, v.size() * sizeof(T)), what);
            cuda_check(cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), what);
        };
        upload(&d_prod, prod, "batch descriptors");
        upload(&d_maps, maps, "batch tensor maps");
        upload(&d_conv_items, conv, "batch conversion items");
        upload(&d_row_items, row_items, "batch row items");
        upload(&d_crt_items, crt_items, "batch CRT items");
        // streams for capture: the main one and one per concurrent class
        const size_t branches = std::max<size_t>(2, std::max(fold_classes.size(), std::max(row_classes.size(), crt_classes.size())) + 1);
        streams.resize(branches);
        events.resize(branches);
        for (auto& s : streams) cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "batch stream");
        for (auto& e : events) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "batch event");
        capture();
    }

    // (Re)build the graph from the current launch shapes.  One warm run outside
    // capture first sets every kernel's shared-memory attribute.
    void capture() {
        if (graph) {
            cudaGraphExecDestroy(graph);
            graph = nullptr;
        }
        enqueue(streams[0]);
        cuda_check(cudaStreamSynchronize(streams[0]), "batch warm-up");
        cudaGraph_t g = nullptr;
        cuda_check(cudaStreamBeginCapture(streams[0], cudaStreamCaptureModeThreadLocal), "batch capture");
        try {
            enqueue(streams[0]);
        } catch (...) {
            cudaStreamEndCapture(streams[0], &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        cuda_check(cudaStreamEndCapture(streams[0], &g), "batch capture end");
        const cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        cuda_check(e, "batch graph instantiate");
    }

    // Device time of one graph run (mean of `reps`).
    double time_us(int reps) {
        cudaEvent_t e0, e1;
        cuda_check(cudaEventCreate(&e0), "batch timing");
        cuda_check(cudaEventCreate(&e1), "batch timing");
        cuda_check(cudaGraphLaunch(graph, streams[0]), "batch timing");
        cuda_check(cudaEventRecord(e0, streams[0]), "batch timing");
        for (int r = 0; r < reps; ++r) cuda_check(cudaGraphLaunch(graph, streams[0]), "batch timing");
        cuda_check(cudaEventRecord(e1, streams[0]), "batch timing");
        cuda_check(cudaEventSynchronize(e1), "batch timing");
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        return 1000.0 * ms / reps;
    }

    // Coordinate descent over the launch shapes, whole-graph time as the objective.
    double tune(int reps) {
        double best = time_us(reps);
        auto attempt = [&](auto apply, auto undo) {
            apply();
            capture();
            const double t = time_us(reps);
            if (t < best) {
                best = t;
                return;
            }
            undo();
            capture();
        };
        for (auto& rc : row_classes)
            for (int k : {2, 3, 4}) {
                const int cur = rc.radix_log;
                if (k == cur || rc.logC < 10) continue;  // the warp kernel's passes are fixed
                attempt([&] { rc.radix_log = k; }, [&] { rc.radix_log = cur; });
            }
        for (int k : {2, 3, 4}) {
            const int old = conv_ctas_per_sm;
            if (k == old || !conv_items) continue;
            attempt([&] { conv_ctas_per_sm = k; }, [&] { conv_ctas_per_sm = old; });
        }
        for (int k : {1, 2}) {
            const bool differs = std::any_of(crt_classes.begin(), crt_classes.end(),
                                             [&](const CrtClass& cc) { return k < k3t_ctas_per_sm(cc.W, 0); });
            const int old = crt_ctas_per_sm;
            if (differs) attempt([&] { crt_ctas_per_sm = k; }, [&] { crt_ctas_per_sm = old; });
        }
        return best;
    }

    void run(cudaStream_t st) {
        cuda_check(cudaGraphLaunch(graph, st), "batch graph launch");
        count_launches((conv_items ? 1 : fold_classes.size()) + row_classes.size() + crt_classes.size());
    }
};

}  // namespace pm

struct pm_batch {
    pm::BatchCore core;
};

extern "C" int pm_batch_create(pm_batch** out, uint32_t count, const uint32_t* n, const uint64_t* const* q,
                               const uint32_t* q_limbs, uint32_t coef_limbs) {
    if (!out || !n || !q || !q_limbs || count == 0) return pm::fail(PM_ERR_INVALID, "NULL argument or empty batch");
    *out = nullptr;
    try {
        auto b = std::make_unique<pm_batch>();
        b->core.build(count, n, q, q_limbs, coef_limbs);
        *out = b.release();
        return PM_OK;
    } catch (const pm::Failure& f) {
        return pm::fail(f.status, f.what());
    } catch (const std::exception& e) {
        return pm::fail(PM_ERR_INVALID, e.what());
    }
}

extern "C" int pm_batch_buffers(pm_batch* batch, uint64_t** a, uint64_t** b, uint64_t** c, uint64_t* offsets) {
    if (!batch) return pm::fail(PM_ERR_INVALID, "NULL batch");
    const auto& s = batch->core;
    if (a) *a = s.d_a;
    if (b) *b = s.d_b;
    if (c) *c = s.d_c;
    if (offsets)
        for (uint32_t z = 0; z < s.count; ++z) offsets[z] = s.io_off[z];
    return PM_OK;
}

extern "C" int pm_batch_copy_in(pm_batch* batch, const uint64_t* a, const uint64_t* b, pm_stream stream) {
    if (!batch || !a || !b) return pm::fail(PM_ERR_INVALID, "NULL argument");
    auto& s = batch->core;
    const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(s.d_a, a, s.io_words * 8, cudaMemcpyDefault, st) != cudaSuccess ||
        cudaMemcpyAsync(s.d_b, b, s.io_words * 8, cudaMemcpyDefault, st) != cudaSuccess)
        return pm::fail(PM_ERR_CUDA, "batch copy in");
    return PM_OK;
}

extern "C" int pm_batch_copy_out(pm_batch* batch, uint64_t* c, pm_stream stream) {
    if (!batch || !c) return pm::fail(PM_ERR_INVALID, "NULL argument");
    auto& s = batch->core;
    if (cudaMemcpyAsync(c, s.d_c, s.io_words * 8, cudaMemcpyDefault, reinterpret_cast<cudaStream_t>(stream)) !=
        cudaSuccess)
        return pm::fail(PM_ERR_CUDA, "batch copy out");
    return PM_OK;
}

extern "C" int pm_batch_run(pm_batch* batch, pm_stream stream) {
    if (!batch) return pm::fail(PM_ERR_INVALID, "NULL batch");
    try {
        batch->core.run(reinterpret_cast<cudaStream_t>(stream));
        return PM_OK;
    } catch (const pm::Failure& f) {
        return pm::fail(f.status, f.what());
    }
}

extern "C" int pm_batch_check(pm_batch* batch) {
    if (!batch) return pm::fail(PM_ERR_INVALID, "NULL batch");
    uint32_t err = 0;
    if (cudaMemcpy(&err, batch->core.d_err, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
        return pm::fail(PM_ERR_CUDA, "read batch error word");
    if (err) {
        cudaMemset(batch->core.d_err, 0, 4);
        return pm::fail(PM_ERR_TIMEOUT, "a tensor-core wait timed out during a batch run");
    }
    return PM_OK;
}

extern "C" int pm_batch_autotune(pm_batch* batch, uint32_t reps, double* us_per_run) {
    if (!batch) return pm::fail(PM_ERR_INVALID, "NULL batch");
    try {
        const double us = batch->core.tune(reps ? int(reps) : 3);
        if (us_per_run) *us_per_run = us;
        return PM_OK;
    } catch (const pm::Failure& f) {
        return pm::fail(f.status, f.what());
    }
}

extern "C" int pm_batch_destroy(pm_batch* batch) {
    delete batch;
    return PM_OK;
}
