// moe_group.cu -- host side of the grouped expert products.
#include "moe_group.h"

#include <algorithm>
#include <cstring>

#include "moe_group.cuh"

using namespace orome;
#define fail orome_fail

bool orome_moe_group_supported(int fmt, uint32_t in_dim) { return (fmt == FMT_Q4_K || fmt == FMT_Q5_K) && in_dim % 256 == 0; }

template <int FMT, bool SWIGLU>
static int launch_group(orome_cuda_ctx *c, const MgArgs &a, cudaStream_t st)
{
    auto kern = moe_group_kernel<FMT, SWIGLU>;
    static int configured[64] = {0};
    if (!configured[c->device]) {
        cudaFuncAttributes fa;
        CU(cudaFuncGetAttributes(&fa, kern));
        const int max_dyn = c->smem_optin - (int)fa.sharedSizeBytes;
        CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn));
        configured[c->device] = max_dyn;
    }
    MgArgs b = a;
    const uint32_t stage = mg_stage_bytes(FMT, a.cap);
    b.nstages = std::min<uint32_t>(MG_MAX_STAGES, (uint32_t)configured[c->device] / stage);
    return orome_launch_pdl_smem(c, "moe_group", kern, dim3(c->sm_count), dim3(MG_THREADS), (size_t)b.nstages * stage, st, b);
}

// Scratch of one call: [pair blocks][order][count] then the records of x and of the activations and the pairs' results.
struct MgScratch {
    size_t blocks, order, count, xq, aq, res, total;      // byte offsets
    MgScratch(size_t T, size_t K, size_t hidden, size_t inter, bool down)
    {
        auto up = [](size_t v) { return (v + 255) / 256 * 256; };
        const size_t n = T * K;
        blocks = 0;
        order = blocks + up(n * sizeof(MgBlock));
        count = order + up(n * 4);
        xq = count + 256;
        aq = xq + up(T * (hidden / 256) * MG_REC);
        res = aq + (down ? up(n * (inter / 256) * MG_REC) : 0);
        total = res + (down ? up(n * hidden * 4) : 0);
    }
};

// A call's scratch.  Two calls may run at the same time -- on two streams, or a replayed graph beside a direct call -- each with
// activations and outputs of its own, so no two of them may share it:
//   direct calls   a piece of the device's pool, allocated and freed in the order of the call's stream (2 + 1 us on the host once
//                  the pool has grown);
//   captured ones  memory of the graph: calls captured on one stream of one capture follow one another in every replay and
//                  share it, and it is used again once the graph and all that was instantiated from it are gone.
struct MgMemory {
    uint8_t *p = nullptr;
    cudaStream_t st;
    bool pooled = false;
    explicit MgMemory(cudaStream_t s) : st(s) {}
    ~MgMemory() { if (pooled) cudaFreeAsync(p, st); }
    MgMemory(const MgMemory &) = delete;
    MgMemory &operator=(const MgMemory &) = delete;
};

static void CUDART_CB graph_scratch_gone(void *flag)
{
    auto *f = static_cast<std::shared_ptr<std::atomic<bool>> *>(flag);
    (*f)->store(true);
    delete f;
}

// OROME_ENOTSUP: no memory, or a capture that cannot own any; the caller has forms that need none.
static int take_memory(orome_cuda_ctx *c, size_t bytes, MgMemory &m)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    CU(cudaStreamGetCaptureInfo(m.st, &cap, &id, &graph, nullptr, nullptr));
    if (cap == cudaStreamCaptureStatusNone) {
        m.p = static_cast<uint8_t *>(orome_pool_alloc(c, bytes, m.st));
        if (!m.p) return OROME_ENOTSUP;
        m.pooled = true;
        return OROME_OK;
    }
    if (cap != cudaStreamCaptureStatusActive) return OROME_ENOTSUP;
    GraphScratch *g = nullptr;
    for (GraphScratch &s : c->graph_scratch)
        if (!s.gone->load() && s.capture == id && s.stream == m.st && s.bytes >= bytes) { m.p = static_cast<uint8_t *>(s.mem); return OROME_OK; }
    for (GraphScratch &s : c->graph_scratch)
        if (!g && s.gone->load() && s.bytes >= bytes) g = &s;
    if (!g) {
        size_t size = 1 << 20;
        while (size < bytes) size *= 2;      // so that later captures of other sizes find it large enough
        // cudaMalloc does not touch the capture, but has to be let through while one is going on
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CU(cudaThreadExchangeStreamCaptureMode(&mode));
        void *p = nullptr;
        const cudaError_t e = cudaMalloc(&p, size);
        CU(cudaThreadExchangeStreamCaptureMode(&mode));
        if (e != cudaSuccess) { (void)cudaGetLastError(); return OROME_ENOTSUP; }
        c->graph_scratch.push_back(GraphScratch{0, nullptr, p, size, std::make_shared<std::atomic<bool>>(true)});
        g = &c->graph_scratch.back();
    }
    auto flag = std::make_shared<std::atomic<bool>>(false);
    auto *held = new std::shared_ptr<std::atomic<bool>>(flag);
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, held, graph_scratch_gone, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        (void)cudaGetLastError();
        delete held;
        return OROME_ENOTSUP;
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        (void)cudaGetLastError();
        cudaUserObjectRelease(obj, 1);
        return OROME_ENOTSUP;
    }
    *g = GraphScratch{id, m.st, g->mem, g->bytes, flag};
    m.p = static_cast<uint8_t *>(g->mem);
    return OROME_OK;
}

int orome_moe_group(orome_cuda_ctx *c, const OromeExpertLayerRef *L, int layout, bool gate_up, bool down, const float *x, int n_tokens, int ldx,
                    const uint32_t *idx, const float *w, uint32_t K, uint32_t hidden, uint32_t inter, float *act, float *out, int ldo, cudaStream_t st)
{
    const uint8_t *base = static_cast<const uint8_t *>(L->buffer);
    const int gfmt = (int)L->gate.format, dfmt = (int)L->down.format;
    constexpr int SLICE = 1024;      // tokens a pass: bounds the pairs' results (64 MiB at a hidden size of 2048)
    const MgScratch most(std::min(n_tokens, SLICE), K, hidden, inter, down);
    MgMemory memory(st);
    int rc = take_memory(c, most.total, memory);
    if (rc) return rc;
    uint8_t *mem = memory.p;
    for (int t0 = 0; t0 < n_tokens; t0 += SLICE) {
        const int T = std::min(n_tokens - t0, SLICE);
        const MgScratch sc(T, K, hidden, inter, down);
        MgArgs a;
        memset(&a, 0, sizeof a);
        // Pairs of an item: 32 where experts have many tokens; 8 vectors a stage leave room for a deeper ring where they
        // have few (a group of more is simply two items).
        a.cap = T * (int)K <= 512 ? 8 : MG_MAX_CAP;
        a.K = K; a.layout = layout; a.status = c->status_dev;
        a.order = reinterpret_cast<uint32_t *>(mem + sc.order);
        a.blocks = reinterpret_cast<MgBlock *>(mem + sc.blocks);
        a.n_blocks = reinterpret_cast<uint32_t *>(mem + sc.count);
        float *act0 = act + (size_t)t0 * K * inter;
        const uint32_t units = hidden / 256, quant = gate_up ? std::min<uint32_t>(((uint32_t)T * units + 31) / 32, 2u * c->sm_count) : 0u;
        rc = orome_launch_pdl(c, "moe_prepare", moe_prepare_kernel, dim3(1 + quant), dim3(1024), st, idx + (size_t)t0 * 8, (uint32_t)T, K, a.cap,
                              reinterpret_cast<uint32_t *>(mem + sc.order), reinterpret_cast<MgBlock *>(mem + sc.blocks),
                              reinterpret_cast<uint32_t *>(mem + sc.count), x + (size_t)t0 * ldx, (uint32_t)ldx, units, mem + sc.xq);
        if (rc) return rc;
        if (gate_up) {
            a.w0 = base + L->gate.offset; a.w1 = base + L->up.offset; a.stride = L->gate.expert_stride;
            a.rows = inter; a.units = units; a.row_bytes = units * mg_unit(gfmt);
            a.xq = mem + sc.xq; a.x_per_token = 1; a.out = act0;
            rc = gfmt == FMT_Q4_K ? launch_group<FMT_Q4_K, true>(c, a, st) : launch_group<FMT_Q5_K, true>(c, a, st);
            if (rc) return rc;
        }
        if (down) {
            const uint32_t aunits = inter / 256;
            rc = orome_launch_pdl(c, "moe_quantize", moe_quantize_kernel, dim3((aunits + 7) / 8, (uint32_t)T * K), dim3(256), st, (const float *)act0, inter, aunits,
                                  mem + sc.aq);
            if (rc) return rc;
            a.w0 = base + L->down.offset; a.w1 = nullptr; a.stride = L->down.expert_stride;
            a.rows = hidden; a.units = aunits; a.row_bytes = aunits * mg_unit(dfmt);
            a.xq = mem + sc.aq; a.x_per_token = 0; a.out = reinterpret_cast<float *>(mem + sc.res);
            rc = dfmt == FMT_Q4_K ? launch_group<FMT_Q4_K, false>(c, a, st) : launch_group<FMT_Q5_K, false>(c, a, st);
            if (rc) return rc;
            rc = orome_launch_pdl(c, "moe_sum", moe_sum_kernel, dim3((hidden + 255) / 256, (uint32_t)T), dim3(256), st, (const float *)(mem + sc.res),
                                  w + (size_t)t0 * 8, K, hidden, out + (size_t)t0 * ldo, (uint32_t)ldo);
            if (rc) return rc;
        }
    }
    return OROME_OK;
}
