// Engine implementation: checkpoint loading, HBM layout, work buffers, the packed forward step.
#include "engine.hpp"

#include <algorithm>
#include <cstring>
#include <mutex>

#include "kernels.cuh"
#include "safetensors.hpp"
#include "rows_linear.cuh"
#include "sample_cluster.cuh"
#include "decode_stream_layout.hpp"
#include "wkv_rows.cuh"
#include "wkv_chunk.cuh"

namespace rsv {

// ------------------------------------------------------------------------------------------------
// launch bookkeeping: every kernel goes through LAUNCH so that it is counted and, when profiling is
// on, timed with a CUDA event pair on the model's stream (PROF_CUDA_KERNEL in the reference,
// src/backend_cuda.rs:412-460).
// ------------------------------------------------------------------------------------------------
struct LaunchScope {
    Model& m;
    const char* name;
    LaunchScope(Model& m_, const char* n) : m(m_), name(n) {
        if (m.prof_on) cudaEventRecord(m.ev0, m.stream);
    }
    ~LaunchScope() {
        ++m.launches;
        if (m.prof_on) {
            cudaEventRecord(m.ev1, m.stream);
            cudaEventSynchronize(m.ev1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, m.ev0, m.ev1);
            auto& p = m.prof[name];
            p.ms += ms;
            p.launches += 1;
        }
    }
};
#define LAUNCH(model, name) if (LaunchScope _ls{model, name}; true)

// Launch with the programmatic-stream-serialization attribute: the kernel may be scheduled while its predecessor in the
// stream is still running and synchronises with it through pdl_wait().  Only kernels that call pdl_wait() before they
// touch anything an earlier kernel of the step produces are launched this way.
template <typename... KArgs, typename... Args>
static void launch_pdl_on(cudaStream_t stream, bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args&&... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    RSV_CUDA(cudaLaunchKernelEx(&cfg, kernel, KArgs(std::forward<Args>(args))...));
}
template <typename... KArgs, typename... Args>
static void launch_pdl(Model& m, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args&&... args) {
    launch_pdl_on(m.stream, m.use_pdl, kernel, grid, block, smem, std::forward<Args>(args)...);
}

// The same as a launch of thread-block clusters of `cluster` CTAs.
template <typename... KArgs, typename... Args>
static void launch_pdl_cluster(Model& m, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int cluster, Args&&... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m.stream;
    cudaLaunchAttribute at[2];
    memset(at, 0, sizeof(at));
    int n = 0;
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster;
    at[n].val.clusterDim.y = 1;
    at[n].val.clusterDim.z = 1;
    ++n;
    if (m.use_pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    RSV_CUDA(cudaLaunchKernelEx(&cfg, kernel, KArgs(std::forward<Args>(args))...));
}

static void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw CudaError(std::string("kernel launch failed (") + what + "): " + cudaGetErrorString(e));
}

// ------------------------------------------------------------------------------------------------
// loading
// ------------------------------------------------------------------------------------------------
namespace {

std::vector<float> to_f32(const StTensor& t) {
    std::vector<float> out((size_t)t.numel());
    if (t.dtype == "F32") {
        if (t.nbytes != out.size() * 4) throw std::runtime_error("tensor byte size mismatch");
        memcpy(out.data(), t.data, t.nbytes);
    } else if (t.dtype == "F16") {
        if (t.nbytes != out.size() * 2) throw std::runtime_error("tensor byte size mismatch");
        const uint16_t* h = (const uint16_t*)t.data;
        for (size_t i = 0; i < out.size(); ++i) out[i] = half_bits_to_float(h[i]);
    } else {
        throw std::runtime_error("unsupported dtype " + t.dtype + " (need F16 or F32)");  // src/model.rs:208-217
    }
    return out;
}

std::vector<uint16_t> to_f16_bits(const StTensor& t) {
    std::vector<uint16_t> out((size_t)t.numel());
    if (t.dtype == "F16") {
        memcpy(out.data(), t.data, out.size() * 2);
    } else if (t.dtype == "F32") {
        const float* f = (const float*)t.data;
        for (size_t i = 0; i < out.size(); ++i) out[i] = float_to_half_bits(f[i]);
    } else {
        throw std::runtime_error("unsupported dtype " + t.dtype + " (need F16 or F32)");
    }
    return out;
}


// cuTensorMapEncodeTiled is fetched through the runtime so that the library does not link libcuda directly.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        RSV_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) throw CudaError("cuTensorMapEncodeTiled is not available in this driver");
        fn = (EncodeTiledFn)p;
    }
    return fn;
}
// 2-D K-major operand [rows, kelems]: box = 128 bytes of K x box_rows rows, 128-byte swizzle.
void encode_kmajor_map(CUtensorMap* map, bool i8, void* base, size_t rows, size_t kelems, int box_rows) {
    const size_t es = i8 ? 1 : 2;
    cuuint64_t dims[2] = {(cuuint64_t)kelems, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(kelems * es)};
    cuuint32_t box[2] = {(cuuint32_t)(kTcKBlockBytes / es), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled_fn()(map, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
}
// All layers' WKV states of a State as one row-major fp32 tensor [rows][64]; box = 32 columns x 64 rows with the 128-byte swizzle.
void encode_state_map(CUtensorMap* map, float* base, size_t rows) {
    cuuint64_t dims[2] = {64, (cuuint64_t)rows};
    cuuint64_t strides[1] = {64 * sizeof(float)};
    cuuint32_t box[2] = {32, 64};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled (state) failed with code " + std::to_string((int)r));
}
inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Loader {
    Model& m;
    const SafeTensorsFile* st;

    void* dev_alloc(size_t bytes) {
        void* p = nullptr;
        RSV_CUDA(device_malloc(&p, std::max<size_t>(bytes, 16)));
        m.allocs.push_back(p);
        m.weight_bytes += bytes;
        return p;
    }
    void* upload(const void* src, size_t bytes) {
        void* p = dev_alloc(bytes);
        RSV_CUDA(cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice));
        return p;
    }
    float* vec(const std::string& key, size_t expect) {
        std::vector<float> v = to_f32(st->get(key));
        if (v.size() != expect) throw std::runtime_error(key + ": expected " + std::to_string(expect) + " elements, file has " + std::to_string(v.size()));
        return (float*)upload(v.data(), v.size() * 4);
    }
    // [out,in] matrix: int8 pair if `{key}.int8_idx` exists (as src/gpu_model.rs:3438-3441), else fp16.
    LinearW linear(const std::string& key, int M, int K) {
        LinearW L;
        L.M = M;
        L.K = K;
        if (st->has(key + ".int8_idx")) {
            const StTensor& it = st->get(key + ".int8_idx");
            const StTensor& zt = st->get(key + ".int8_sz");
            if (K % 128) throw std::runtime_error(key + ": int8 needs K % 128 == 0");
            if (it.dtype != "U8" || it.nbytes != (size_t)M * K) throw std::runtime_error(key + ".int8_idx: expected U8 [" + std::to_string(M) + "," + std::to_string(K) + "]");
            if (zt.dtype != "U32" || zt.nbytes != (size_t)M * (K / 128) * 4) throw std::runtime_error(key + ".int8_sz: expected U32 [M, K/128]");
            L.wtype = W_INT8;
            L.w = upload(it.data, it.nbytes);
            L.sz = (uint32_t*)upload(zt.data, zt.nbytes);
            prepare_tc_i8(L, (const uint32_t*)zt.data);
        } else {
            const StTensor& t = st->get(key);
            if (t.numel() != (int64_t)M * K) throw std::runtime_error(key + ": shape mismatch");
            if (K % 8) throw std::runtime_error(key + ": fp16 needs K % 8 == 0");
            L.wtype = W_F16;
            if (t.dtype == "F16") {
                L.w = upload(t.data, t.nbytes);
                prepare_tc_f16(L);
            } else {
                auto h = to_f16_bits(t);
                L.w = upload(h.data(), h.size() * 2);
                prepare_tc_f16(L);
            }
        }
        return L;
    }
    // int8: files with one (scale, zero) per output row (all groups of a row equal) keep them as two vectors; others keep the words
    // transposed, so that the 128 output rows of a tile read a group's words together.
    void prepare_tc_i8(LinearW& L, const uint32_t* sz_host) {
        const int KG = L.K / 128;
        bool per_row = true;
        for (int m = 0; m < L.M && per_row; ++m)
            for (int g = 1; g < KG && per_row; ++g) per_row = sz_host[(size_t)m * KG + g] == sz_host[(size_t)m * KG];
        if (per_row) {
            std::vector<float> sc(L.M), zr(L.M);
            for (int m = 0; m < L.M; ++m) {
                sc[m] = half_bits_to_float((uint16_t)(sz_host[(size_t)m * KG] & 0xFFFFu));
                zr[m] = half_bits_to_float((uint16_t)(sz_host[(size_t)m * KG] >> 16));
            }
            L.wscale = (float*)upload(sc.data(), sc.size() * 4);
            L.wzero = (float*)upload(zr.data(), zr.size() * 4);
        } else {
            std::vector<uint32_t> t((size_t)KG * L.M);
            for (int m = 0; m < L.M; ++m)
                for (int g = 0; g < KG; ++g) t[(size_t)g * L.M + m] = sz_host[(size_t)m * KG + g];
            L.szt = (uint32_t*)upload(t.data(), t.size() * 4);
        }
        encode_kmajor_map(&L.amap, true, L.w, L.M, L.K, kTcTileM);
    }
    void prepare_tc_f16(LinearW& L) {
        encode_kmajor_map(&L.amap, false, L.w, L.M, L.K, kTcTileM);  // boxes past the matrix read zeros
    }
    // Low-rank pair member.  The file holds either [in,out] or [out,in] (src/model.rs:564-581 accepts
    // both, first match wins when in == out); HBM always holds [out,in] fp16.
    LinearW lowrank(const std::string& key, int in_dim, int out_dim) {
        const StTensor& t = st->get(key);
        if (t.shape.size() != 2) throw std::runtime_error(key + ": expected a 2-D tensor");
        std::vector<uint16_t> h = to_f16_bits(t);
        std::vector<uint16_t> oi((size_t)in_dim * out_dim);
        if (t.shape[0] == in_dim && t.shape[1] == out_dim) {
            for (int i = 0; i < in_dim; ++i)
                for (int o = 0; o < out_dim; ++o) oi[(size_t)o * in_dim + i] = h[(size_t)i * out_dim + o];
        } else if (t.shape[0] == out_dim && t.shape[1] == in_dim) {
            oi = h;
        } else {
            throw std::runtime_error(key + ": unexpected shape, want [" + std::to_string(in_dim) + "," + std::to_string(out_dim) + "] or its transpose");
        }
        if (in_dim % 8) throw std::runtime_error(key + ": inner dimension must be a multiple of 8");
        LinearW L;
        L.M = out_dim;
        L.K = in_dim;
        L.wtype = W_F16;
        L.w = upload(oi.data(), oi.size() * 2);
        prepare_tc_f16(L);
        return L;
    }
};

}  // namespace

std::unique_ptr<Model> Model::load(const std::string& path, int device) {
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0)
        throw CudaError(std::string("no CUDA device available (") + cudaGetErrorString(e) + "): this library has no CPU fallback");
    if (device < 0 || device >= ndev) throw std::runtime_error("device index out of range");
    RSV_CUDA(cudaSetDevice(device));
    cudaDeviceProp prop;
    RSV_CUDA(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10) throw std::runtime_error("this library is built for sm_100a (B200) only; device is sm_" + std::to_string(prop.major) + std::to_string(prop.minor));

    SafeTensorsFile st(path);
    auto m = std::make_unique<Model>();
    m->device = device;
    m->state_pool = std::make_shared<StatePool>(device);
    Config& c = m->cfg;
    // hyper-parameters come from tensor shapes only (src/gpu_model.rs:406-444)
    int max_layer = -1;
    for (auto& kv : st.tensors()) {
        const std::string& k = kv.first;
        if (k.rfind("blocks.", 0) == 0) {
            size_t p = k.find('.', 7);
            if (p != std::string::npos) {
                bool digits = p > 7;
                for (size_t i = 7; i < p; ++i) digits = digits && k[i] >= '0' && k[i] <= '9';
                if (digits) max_layer = std::max(max_layer, std::stoi(k.substr(7, p - 7)));
            }
        }
    }
    if (max_layer < 0) throw std::runtime_error("no blocks.* tensors in checkpoint");
    c.n_layer = max_layer + 1;
    const StTensor& emb = st.get("emb.weight");
    if (emb.shape.size() != 2) throw std::runtime_error("emb.weight must be 2-D");
    c.vocab = (int)emb.shape[0];
    c.n_embd = (int)emb.shape[1];
    const StTensor& rk = st.get("blocks.0.att.r_k");
    if (rk.shape.size() != 2) throw std::runtime_error("blocks.0.att.r_k must be [H,N]");
    c.n_head = (int)rk.shape[0];
    c.head_size = (int)rk.shape[1];
    auto mid_of = [&](const char* k) {
        const StTensor& t = st.get(k);
        if (t.shape.size() != 2) throw std::runtime_error(std::string(k) + " must be 2-D");
        return (int)(t.shape[0] == c.n_embd ? t.shape[1] : t.shape[0]);
    };
    c.w_mid = mid_of("blocks.0.att.w1");
    c.a_mid = mid_of("blocks.0.att.a1");
    c.v_mid = mid_of("blocks.0.att.v1");
    c.g_mid = mid_of("blocks.0.att.g1");
    c.ffn_hidden = (int)(st.has("blocks.0.ffn.key.weight") ? st.get("blocks.0.ffn.key.weight").shape.at(0)
                                                            : st.get("blocks.0.ffn.key.weight.int8_idx").shape.at(0));
    if (c.head_size != kHeadSize) throw std::runtime_error("head_size must be 64");
    if (c.n_head * c.head_size != c.n_embd) throw std::runtime_error("n_head * head_size != n_embd");
    if (c.n_embd % 8 || c.ffn_hidden % 8) throw std::runtime_error("n_embd and ffn_hidden must be multiples of 8");

    m->num_sms = prop.multiProcessorCount;
    if (const char* e = getenv("RSV_NO_STREAM"))
        if (*e && *e != '0') m->use_stream = false;
    if (const char* e = getenv("RSV_NO_GRAPH"))
        if (*e && *e != '0') m->use_graphs = false;
    if (const char* e = getenv("RSV_NO_PDL"))
        if (*e && *e != '0') m->use_pdl = false;
    RSV_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    RSV_CUDA(cudaEventCreate(&m->ev0));
    RSV_CUDA(cudaEventCreate(&m->ev1));
    RSV_CUDA(cudaEventCreate(&m->tev[0]));
    RSV_CUDA(cudaEventCreate(&m->tev[1]));

    Loader ld{*m, &st};
    const int C = c.n_embd, F = c.ffn_hidden;
    {
        auto h = to_f16_bits(emb);
        m->emb = (__half*)ld.upload(h.data(), h.size() * 2);
    }
    m->ln0_w = ld.vec("blocks.0.ln0.weight", C);
    m->ln0_b = ld.vec("blocks.0.ln0.bias", C);
    m->ln_out_w = ld.vec("ln_out.weight", C);
    m->ln_out_b = ld.vec("ln_out.bias", C);
    m->head = ld.linear("head.weight", c.vocab, C);
    m->layers.resize(c.n_layer);
    for (int i = 0; i < c.n_layer; ++i) {
        const std::string p = "blocks." + std::to_string(i) + ".";
        LayerW& L = m->layers[i];
        L.ln1_w = ld.vec(p + "ln1.weight", C);
        L.ln1_b = ld.vec(p + "ln1.bias", C);
        L.ln2_w = ld.vec(p + "ln2.weight", C);
        L.ln2_b = ld.vec(p + "ln2.bias", C);
        L.lnx_w = ld.vec(p + "att.ln_x.weight", C);
        L.lnx_b = ld.vec(p + "att.ln_x.bias", C);
        L.x_r = ld.vec(p + "att.x_r", C);
        L.x_w = ld.vec(p + "att.x_w", C);
        L.x_k = ld.vec(p + "att.x_k", C);
        L.x_v = ld.vec(p + "att.x_v", C);
        L.x_a = ld.vec(p + "att.x_a", C);
        L.x_g = ld.vec(p + "att.x_g", C);
        L.ffn_x_k = ld.vec(p + "ffn.x_k", C);
        L.w0 = ld.vec(p + "att.w0", C);
        L.a0 = ld.vec(p + "att.a0", C);
        L.v0 = ld.vec(p + "att.v0", C);
        L.r_k = ld.vec(p + "att.r_k", C);
        L.k_k = ld.vec(p + "att.k_k", C);
        L.k_a = ld.vec(p + "att.k_a", C);
        L.Wr = ld.linear(p + "att.receptance.weight", C, C);
        L.Wk = ld.linear(p + "att.key.weight", C, C);
        L.Wv = ld.linear(p + "att.value.weight", C, C);
        L.Wo = ld.linear(p + "att.output.weight", C, C);
        L.Wfk = ld.linear(p + "ffn.key.weight", F, C);
        L.Wfv = ld.linear(p + "ffn.value.weight", C, F);
        L.w1 = ld.lowrank(p + "att.w1", C, c.w_mid);
        L.w2 = ld.lowrank(p + "att.w2", c.w_mid, C);
        L.a1 = ld.lowrank(p + "att.a1", C, c.a_mid);
        L.a2 = ld.lowrank(p + "att.a2", c.a_mid, C);
        L.v1 = ld.lowrank(p + "att.v1", C, c.v_mid);
        L.v2 = ld.lowrank(p + "att.v2", c.v_mid, C);
        L.g1 = ld.lowrank(p + "att.g1", C, c.g_mid);
        L.g2 = ld.lowrank(p + "att.g2", c.g_mid, C);
    }
    auto same_formats = [&](const LayerW& a, const LayerW& b) {
        const auto x = a.big(), y = b.big();
        bool same = true;
        for (size_t i = 0; i < x.size(); ++i) same = same && x[i]->wtype == y[i]->wtype && x[i]->row_scaled() == y[i]->row_scaled();
        return same;
    };
    for (int i = 0; i < c.n_layer; ++i)
        if (std::none_of(m->format_layers.begin(), m->format_layers.end(), [&](int j) { return same_formats(m->layers[j], m->layers[i]); })) m->format_layers.push_back(i);
    m->pinned_bytes = 1 << 18;
    RSV_CUDA(cudaMallocHost(&m->pinned, m->pinned_bytes * Model::kPinRing));
    for (int i = 0; i < Model::kPinRing; ++i) RSV_CUDA(cudaEventCreateWithFlags(&m->pin_ev[i], cudaEventDisableTiming));
    RSV_CUDA(device_malloc(&m->ws.status, 2 * sizeof(int)));
    RSV_CUDA(device_malloc(&m->ws.tok_pos, sizeof(int)));
    RSV_CUDA(cudaMemsetAsync(m->ws.status, 0, 2 * sizeof(int), m->stream));
    RSV_CUDA(cudaMemsetAsync(m->ws.tok_pos, 0, sizeof(int), m->stream));
    return m;
}

std::unique_ptr<Model> Model::create_bare(int device) {
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0)
        throw CudaError(std::string("no CUDA device available (") + cudaGetErrorString(e) + "): this library has no CPU fallback");
    if (device < 0 || device >= ndev) throw std::runtime_error("device index out of range");
    RSV_CUDA(cudaSetDevice(device));
    cudaDeviceProp prop;
    RSV_CUDA(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10) throw std::runtime_error("this library is built for sm_100a (B200) only");
    auto m = std::make_unique<Model>();
    m->device = device;
    m->state_pool = std::make_shared<StatePool>(device);
    m->num_sms = prop.multiProcessorCount;
    RSV_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    RSV_CUDA(cudaEventCreate(&m->ev0));
    RSV_CUDA(cudaEventCreate(&m->ev1));
    RSV_CUDA(cudaEventCreate(&m->tev[0]));
    RSV_CUDA(cudaEventCreate(&m->tev[1]));
    RSV_CUDA(device_malloc(&m->ws.status, 2 * sizeof(int)));
    RSV_CUDA(cudaMemsetAsync(m->ws.status, 0, 2 * sizeof(int), m->stream));
    return m;
}

static void free_workspace(Workspace& w) {
    void* ptrs[] = {w.x, w.x2, w.delta, w.r, w.k, w.v, w.w, w.a, w.g, w.yg, w.xb, w.mid, w.h, w.vfirst, w.logits, w.staging_t, w.staging_c, w.ymax, w.hmax, w.tokens, w.row_meta, w.seg_meta, w.out_rows, w.samp_temp, w.samp_cnt};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    int* status = w.status;
    int* pos = w.tok_pos;
    Workspace keep = w;
    w = Workspace{};
    w.status = status;
    w.tok_pos = pos;
    w.tok_list = keep.tok_list;
    w.tok_list_cap = keep.tok_list_cap;
    w.op_mem = keep.op_mem;
    w.op_bytes = keep.op_bytes;
    w.wkv_tmp = keep.wkv_tmp;
}

Model::~Model() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    if (state_pool) state_pool->release(true);
    free_workspace(ws);
    if (ws.status) cudaFree(ws.status);
    if (ws.tok_pos) cudaFree(ws.tok_pos);
    if (ws.tok_list) cudaFree(ws.tok_list);
    for (void* p : allocs) cudaFree(p);
    if (ws.op_mem) cudaFree(ws.op_mem);
    ws.wkv_tmp.release();
    for (void* p : {sctx.d_layers, sctx.wstream, sctx.hstream, (void*)sctx.exchange, (void*)sctx.cand_val, (void*)sctx.cand_idx, (void*)sctx.grid_bar})
        if (p) cudaFree(p);
    if (pinned) cudaFreeHost(pinned);
    if (pinned_out) cudaFreeHost(pinned_out);
    for (cudaEvent_t e : out_ev)
        if (e) cudaEventDestroy(e);
    for (int i = 0; i < kPinRing; ++i)
        if (pin_ev[i]) cudaEventDestroy(pin_ev[i]);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (tev[0]) cudaEventDestroy(tev[0]);
    if (tev[1]) cudaEventDestroy(tev[1]);
    if (stream) cudaStreamDestroy(stream);
}

State::~State() {
    if (!wkv) return;
    cudaSetDevice(pool->device);
    pool->give(bytes, wkv);
}

void State::allocate(Model* m, int64_t slots) {
    model = m;
    cap = slots;
    const Config& c = m->cfg;
    auto aligned = [](size_t floats) { return (floats + 63) / 64 * 64; };
    const size_t nx = aligned((size_t)c.n_layer * cap * c.n_embd), ns = aligned((size_t)c.n_layer * cap * c.n_head * kHeadSize * kHeadSize);
    bytes = (ns + 2 * nx + (size_t)cap * c.n_embd) * 4;
    pool = m->state_pool;
    wkv = pool->take(bytes);
    if (!wkv) {
        float* p = nullptr;
        RSV_CUDA(device_malloc(&p, bytes));
        wkv = p;
    }
    tmix_x = wkv + ns;
    cmix_x = tmix_x + nx;
    v_first = cmix_x + nx;
}

void State::clear() { RSV_CUDA(cudaMemsetAsync(wkv, 0, bytes, model->stream)); }

void Model::ensure_workspace(int rows, int outs, int segs) {
    if (rows <= ws.rows && outs <= ws.outs && segs <= ws.segs) return;
    RSV_CUDA(cudaStreamSynchronize(stream));
    // Growing frees and reallocates every array (each a device synchronisation), so a dimension that grows a second time gets
    // a quarter of slack: a server whose step size creeps up reallocates a few times, not at every new maximum.
    auto grow = [](int want, int have) { return want <= have ? have : (have > 1 ? want + want / 4 : want); };
    rows = grow(rows, ws.rows);
    outs = grow(outs, ws.outs);
    segs = grow(segs, ws.segs);
    free_workspace(ws);
    const size_t C = cfg.n_embd, F = cfg.ffn_hidden, V = cfg.vocab, R = rows;
    auto fa = [&](float*& p, size_t n) { RSV_CUDA(device_malloc(&p, std::max<size_t>(n, 4) * sizeof(float))); };
    fa(ws.x, R * C);
    fa(ws.x2, R * C);
    fa(ws.delta, R * C);
    fa(ws.r, R * C);
    fa(ws.k, R * C);
    fa(ws.v, R * C);
    fa(ws.w, R * C);
    fa(ws.a, R * C);
    fa(ws.g, R * C);
    fa(ws.yg, R * C);
    fa(ws.xb, R * C);
    fa(ws.mid, R * (size_t)cfg.mids());
    fa(ws.h, R * F);
    fa(ws.vfirst, R * C);
    fa(ws.logits, (size_t)outs * V);
    fa(ws.ymax, R * 2 * (size_t)cfg.n_head);
    fa(ws.hmax, R * ((F + kRlTileM - 1) / kRlTileM));
    fa(ws.staging_t, (size_t)segs * C);
    fa(ws.staging_c, (size_t)segs * C);
    if (V > (size_t)kScMaxV) {  // the sampler of smaller vocabularies needs no work area
        fa(ws.samp_temp, (size_t)outs * V);
        RSV_CUDA(device_malloc(&ws.samp_cnt, std::max<size_t>((size_t)outs * V, 4) * sizeof(uint32_t)));
    }
    RSV_CUDA(device_malloc(&ws.tokens, R * sizeof(uint32_t)));
    RSV_CUDA(cudaMemsetAsync(ws.tokens, 0, R * sizeof(uint32_t), stream));
    RSV_CUDA(device_malloc(&ws.row_meta, R * sizeof(RowMeta)));
    RSV_CUDA(device_malloc(&ws.seg_meta, (size_t)segs * sizeof(SegMeta)));
    RSV_CUDA(device_malloc(&ws.out_rows, (size_t)std::max(outs, 1) * sizeof(int)));
    const size_t need = R * sizeof(RowMeta) + (size_t)segs * sizeof(SegMeta) + (size_t)outs * sizeof(int) + R * sizeof(uint32_t) + 256;
    if (need > pinned_bytes) {
        cudaFreeHost(pinned);
        pinned = nullptr;
        pinned_bytes = 0;
        RSV_CUDA(cudaMallocHost(&pinned, need * 2 * kPinRing));
        pinned_bytes = need * 2;
    }
    ws.rows = rows;  // (last: an allocation that failed leaves a workspace of no rows)
    ws.outs = outs;
    ws.segs = segs;
}

void Model::ensure_pinned_out(size_t bytes) {
    for (cudaEvent_t& e : out_ev)
        if (!e) RSV_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if (bytes <= pinned_out_bytes) return;
    if (pinned_out) cudaFreeHost(pinned_out);
    pinned_out = nullptr;
    pinned_out_bytes = 0;
    RSV_CUDA(cudaMallocHost(&pinned_out, bytes));
    pinned_out_bytes = bytes;
}

void Model::upload_plan(const StepPlan& plan) {
    const int R = (int)plan.rows.size(), S = (int)plan.segs.size(), O = (int)plan.out_rows.size();
    ensure_workspace(R, std::max(O, 1), S);
    // next area of the staging ring; its previous copies (kPinRing uploads ago) must have completed
    const int slot = pin_next;
    pin_next = (pin_next + 1) % kPinRing;
    if (pin_ev[slot]) RSV_CUDA(cudaEventSynchronize(pin_ev[slot]));
    char* p = (char*)pinned + (size_t)slot * pinned_bytes;
    memcpy(p, plan.rows.data(), R * sizeof(RowMeta));
    RSV_CUDA(cudaMemcpyAsync(ws.row_meta, p, R * sizeof(RowMeta), cudaMemcpyHostToDevice, stream));
    p += R * sizeof(RowMeta);
    SegMeta* sm = reinterpret_cast<SegMeta*>(p);
    for (int i = 0, chunks = 0; i < S; ++i) {
        sm[i] = plan.segs[i];
        sm[i].chunk0 = chunks;
        chunks += wkv_chunks_of(sm[i].len);
    }
    RSV_CUDA(cudaMemcpyAsync(ws.seg_meta, p, S * sizeof(SegMeta), cudaMemcpyHostToDevice, stream));
    p += S * sizeof(SegMeta);
    if (O) {
        memcpy(p, plan.out_rows.data(), O * sizeof(int));
        RSV_CUDA(cudaMemcpyAsync(ws.out_rows, p, O * sizeof(int), cudaMemcpyHostToDevice, stream));
    }
    if (pin_ev[slot]) RSV_CUDA(cudaEventRecord(pin_ev[slot], stream));
}

// ------------------------------------------------------------------------------------------------
// linear launch helper
// ------------------------------------------------------------------------------------------------
namespace {

template <int RT>
void launch_linear_rt(Model& m, const LinProb& P, int nblk, int R, size_t smem) {
    static bool configured[8] = {false};
    int dev = m.device & 7;
    if (!configured[dev]) {
        RSV_CUDA(cudaFuncSetAttribute(linear_rows_kernel<RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured[dev] = true;
    }
    dim3 grid(nblk, (R + RT - 1) / RT);
    linear_rows_kernel<RT><<<grid, kLinWarps * 32, smem, m.stream>>>(P, R);
    check_launch("linear_rows");
}

void run_linear_simt(Model& m, const char* name, const LinearW& W, const float* x, float* y, int R) {
    LinProb P;
    memset(&P, 0, sizeof(P));
    P.w = W.w;
    P.sz = W.sz;
    P.x = x;
    P.y = y;
    P.M = W.M;
    P.K = W.K;
    P.wtype = W.wtype;
    // rows per CTA: aim for a few waves over 148 SMs, but amortise the x staging
    const int unit = kLinWarps * kLinWR;
    P.rows_per_blk = std::min(std::max((W.M / (148 * 4)) / unit * unit, unit), 8 * unit);
    const int blk = (W.M + P.rows_per_blk - 1) / P.rows_per_blk;
    auto smem_for = [&](int rt) { return (size_t)rt * W.K * 4 + (W.wtype == W_INT8 ? (size_t)rt * (W.K / 16) * 4 : 0); };
    int rt = R >= 4 ? 4 : (R >= 2 ? 2 : 1);
    while (rt > 1 && smem_for(rt) > 200 * 1024) rt >>= 1;
    if (smem_for(rt) > 200 * 1024) throw std::runtime_error("linear: inner dimension too large for the shared-memory tile");
    LAUNCH(m, name) {
        if (rt == 4)
            launch_linear_rt<4>(m, P, blk, R, smem_for(4));
        else if (rt == 2)
            launch_linear_rt<2>(m, P, blk, R, smem_for(2));
        else
            launch_linear_rt<1>(m, P, blk, R, smem_for(1));
    }
}


// ---- tensor-core path ---------------------------------------------------------------------------
int rl_fmt(const LinearW& W) { return W.wtype != W_INT8 ? RL_F16 : W.row_scaled() ? RL_I8 : RL_I8G; }

// Carves a step's operands out of one block of device memory.
struct OperandCarver {
    uint8_t* base = nullptr;
    size_t used = 0;
    template <typename T>
    T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base + used);
        used += round_up(n * sizeof(T), 1024);
        return p;
    }
    RlOperandOut operand(const RowTiles& t, int fmt, int K, const float* mix = nullptr, int tparts = 1) {
        RlOperandOut o;
        memset(&o, 0, sizeof(o));
        o.mix = mix;
        o.fmt = fmt;
        o.nt = t.nt(fmt);
        o.kblocks = (K + rl_kelems(fmt) - 1) / rl_kelems(fmt);
        o.img = take<uint8_t>(t.image_bytes(fmt, K));
        o.xscale = take<float>((size_t)t.R);
        o.tparts = tparts;
        if (fmt == RL_I8) o.tsum = take<long long>((size_t)t.R * tparts);
        if (fmt == RL_I8G) o.tgrp = take<float>((size_t)t.R * o.kblocks);
        return o;
    }
};
void ensure_operand_memory(Model& m, size_t bytes) {
    Workspace& w = m.ws;
    if (bytes <= w.op_bytes) return;
    RSV_CUDA(cudaStreamSynchronize(m.stream));
    if (w.op_mem) cudaFree(w.op_mem);
    w.op_mem = nullptr;
    w.op_bytes = 0;
    const size_t nb = bytes + bytes / 4;
    RSV_CUDA(device_malloc(&w.op_mem, nb));
    RSV_CUDA(cudaMemsetAsync(w.op_mem, 0, nb, m.stream));
    w.op_bytes = nb;
}

// One linear layer of a launch.  Its operand is a prepared image (`op`), or fp32 activations the kernel converts itself.
struct RlReq {
    const LinearW* W;
    const RlOperandOut* op;
    float* y;
    int ldy;
    int epi;
    const float* bias = nullptr;
    float* y2 = nullptr;
    float* ymax = nullptr;
    const float* x = nullptr;  // op == nullptr: activations [R, ldx]
    int ldx = 0;
};

constexpr size_t kRlRingMax = 196 * 1024;  // stages of the persistent kernel, which has its SM to itself
constexpr size_t kRlHalfSm = 109 * 1024;  // dynamic shared memory of a CTA that leaves room for a second one on its SM

// Bytes of shared memory in which the CTAs of a split tile receive each other's partial sums.
size_t rl_recv_bytes(int rt, int split) { return (size_t)split * ((rt + split - 1) / split) * kRlTileM * 8; }
// How many CTAs share a tile's K.  The step's launches are short (few tiles, weights prefetched behind the previous kernel), so a
// launch wants about one CTA per half SM and few K blocks per CTA, but no second wave.  A split tile of more than 108 rows (fp16) takes a
// whole SM, for the partial sums it receives; counted as half of one, r, k, v and rank projections of 256 rows (132 tiles, 2560 channels)
// went out as two waves of 264 CTAs in 51 us, 33 unsplit.
int rl_split(const Model& m, int jobs, int kb_min, int kb_max, int rt) {
    auto slots = [&](int s) { return rl_recv_bytes(rt, s) + 1024 <= kRlHalfSm ? 2 * m.num_sms : m.num_sms; };
    int s = 1;
    while (s < kRlMaxSplit && 2 * s <= kb_min && jobs * 2 * s <= slots(2 * s) && kb_max / s > 5) s *= 2;
    return s;
}

template <bool GROUPED, bool BUILD>
void rl_launch(Model& m, const char* name, const RlLaunch& L, int ctas, size_t smem) {
    static bool configured[16] = {false};
    if (!configured[m.device & 15]) {
        RSV_CUDA(cudaFuncSetAttribute(rows_linear_kernel<GROUPED, BUILD>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured[m.device & 15] = true;
    }
    LAUNCH(m, name) {
        launch_pdl_cluster(m, rows_linear_kernel<GROUPED, BUILD>, dim3(ctas), dim3(kRlThreads), smem, L.split, L);
        check_launch("rows_linear");
    }
}

template <int WARPS>
void rl_launch_persistent(Model& m, const char* name, const RlLaunch& L, int jobs, size_t smem) {
    static bool configured[16] = {false};
    if (!configured[m.device & 15]) {
        RSV_CUDA(cudaFuncSetAttribute(rows_linear_persistent_kernel<WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRlRingMax + 1024));
        configured[m.device & 15] = true;
    }
    LAUNCH(m, name) {
        launch_pdl(m, rows_linear_persistent_kernel<WARPS>, dim3(std::min(jobs, m.num_sms)), dim3(rl_persistent_threads(WARPS)), smem, L, jobs);
        check_launch("rows_linear_persistent");
    }
}

void run_rows_linear(Model& m, const char* name, const RlReq* reqs, int n, const RowTiles& t) {
    if (n < 1 || n > kRlMaxProb) throw std::runtime_error("rows_linear: too many problems in one launch");
    {
        // The kernel is compiled for one kind of int8 weights.  Matrices with a (scale, zero) per row next to others with one per group
        // (a per-group file in which some rows happen to be uniform) go out in a launch of their own.
        RlReq per_row[kRlMaxProb], rest[kRlMaxProb];
        int nrow = 0, nrest = 0;
        bool mixed = false;
        for (int i = 0; i < n; ++i) {
            if (rl_fmt(*reqs[i].W) == RL_I8)
                per_row[nrow++] = reqs[i];
            else
                rest[nrest++] = reqs[i];
            mixed = mixed || rl_fmt(*reqs[i].W) == RL_I8G;
        }
        if (mixed && nrow) {
            run_rows_linear(m, name, per_row, nrow, t);
            return run_rows_linear(m, name, rest, nrest, t);
        }
    }
    RlLaunch L;
    memset(&L, 0, sizeof(L));
    const bool build = reqs[0].op == nullptr;
    bool grouped = false, row8 = false;
    int jobs = 0, kb_min = 1 << 30, kb_max = 0, nt_max = 0;
    for (int i = 0; i < n; ++i) {
        const RlReq& q = reqs[i];
        const LinearW& W = *q.W;
        RlProb& P = L.p[i];
        P.fmt = rl_fmt(W);
        grouped = grouped || P.fmt == RL_I8G;
        row8 = row8 || P.fmt == RL_I8;
        if ((q.op == nullptr) != build) throw std::runtime_error("rows_linear: prepared and unprepared operands in one launch");
        if (q.op) {
            P.bimg = q.op->img;
            P.xscale = q.op->xscale;
            P.tsum = q.op->tsum;
            P.tgrp = q.op->tgrp;
            P.tparts = q.op->tparts;
        }
        P.wscale = W.wscale;
        P.wzero = W.wzero;
        P.szt = W.szt;
        P.x = q.x;
        P.y = q.y;
        P.y2 = q.y2;
        P.bias = q.bias;
        P.ymax = q.ymax;
        P.ldx = q.ldx;
        P.ldy = q.ldy;
        P.epi = q.epi;
        P.M = W.M;
        P.K = W.K;
        P.kblocks = (W.K + rl_kelems(P.fmt) - 1) / rl_kelems(P.fmt);
        P.job0 = jobs;
        L.amap[i] = W.amap;
        jobs += (W.M + kRlTileM - 1) / kRlTileM * t.n;
        kb_min = std::min(kb_min, P.kblocks);
        kb_max = std::max(kb_max, P.kblocks);
        nt_max = std::max(nt_max, t.nt(P.fmt));
    }
    if (grouped && t.rt > kRlMaxRowsG) throw std::runtime_error("rows_linear: row tile too large for per-group weights");
    L.nprob = n;
    L.R = t.R;
    L.rt = t.rt;
    L.n_tiles = t.n;
    L.nt8 = t.nt8;
    L.nt16 = t.nt16;
    L.status = m.ws.status;
    L.split = build || t.turns ? 1 : rl_split(m, jobs, kb_min, kb_max, t.rt);  // a kernel that builds its operands has to see whole rows
    while ((1 << L.log_split) < L.split) ++L.log_split;
    int nk = 0;
    for (int i = 0; i < n; ++i) nk = std::max(nk, (L.p[i].kblocks + L.split - 1) / L.split);
    // Several full row tiles that fill the GPU without splitting K: the persistent kernel.  Not for tiles of fewer than 16 K blocks, which are all epilogue: the rank
    // back-projections take 8.7 us at 128 rows with a CTA per tile and 13.8 persistent, 13.8 and 14.1 at 256, 15.9 and 16.0 at 384; from four turns on persistent is the
    // faster one, 21.8 and 19.8 at 512 rows, 38.6 and 32.9 at 1024, and so it is with the tiles of 32 rows of per-group files, 16.0 and 14.0 at 256 rows, 27.4 and 23.9 at 512, 50.6
    // and 44.7 at 1024; nor for fp16 tiles of 64 rows that were not cut for turns: they
    // leave half of the matrix instruction's columns out.  One row tile and more weight tiles than two CTAs per SM take at once (the vocabulary head: 512 of them, 336 MB):
    // the second set of CTAs would start its ring from nothing; 3 rows 75 us, persistent 56, 64 rows 83 and 63.
    if (!build && !grouped && (t.turns || (kb_max <= 8 && jobs >= 4 * m.num_sms) || (L.split == 1 && kb_min >= 16 && (t.n > 1 ? row8 || t.rt > kRlMaxRows : jobs > 2 * m.num_sms)))) {
        const size_t st = kRlABytes + (size_t)nt_max * 128;
        L.nt_max = nt_max;
        L.ring = (int)(std::min<size_t>(kRlMaxStages, kRlRingMax / st) * st);
        L.tmem_cols = 64;
        while (L.tmem_cols < 2 * nt_max) L.tmem_cols *= 2;
        const size_t bytes = L.ring + 1024;
        // Several narrow tiles of few rows: eight epilogue warps keep up with the products, and beside sixteen (46 of 64 K registers) the CTAs of the next kernel, which
        // converts the outputs of up to 118 rows, would not all be resident early (a layer of 72 int8 rows, 2560 channels: 112.0 us with sixteen, 110.4 with
        // eight; 112 rows 140.4 and 138.1, 128 the same, 160 rows 166.2 and 168.8).
        if (t.n > 1 && t.R <= 2 * kRlMaxRows)
            rl_launch_persistent<8>(m, name, L, jobs, bytes);
        else
            rl_launch_persistent<16>(m, name, L, jobs, bytes);
        return;
    }
    const size_t stage = kRlABytes + (build ? 0 : (size_t)nt_max * 128), bbuf = build ? (size_t)nk * nt_max * 128 : 0, tg = grouped ? round_up(((size_t)nk * rl_group_rows(t.rt) + kRlMaxRowsG) * 4, 16) : 0;  // (sums of rows past the end are read)
    const size_t recv = L.split > 1 || grouped ? rl_recv_bytes(t.rt, L.split) : 0;  // partial sums reuse the ring
    int stages = std::min(nk, kRlMaxStages);
    while (stages > 2 && stages * stage + bbuf + tg + 1024 > kRlHalfSm) --stages;
    L.ring = (int)std::max(stages * stage, round_up(recv, 1024));
    const size_t smem = L.ring + bbuf + tg + 1024;
    if (smem > 200 * 1024) throw std::runtime_error("rows_linear: operands do not fit in shared memory");
    int cols = 32;
    while (cols < std::max(grouped ? 2 * rl_group_cols(t.nt8) : 0, nt_max)) cols *= 2;
    L.tmem_cols = cols;
    if (build)
        rl_launch<false, true>(m, name, L, jobs, smem);
    else if (grouped)
        rl_launch<true, false>(m, name, L, jobs * L.split, smem);
    else
        rl_launch<false, false>(m, name, L, jobs * L.split, smem);
}

// Short fp16 rows (the rank-space vectors) of few sessions are converted inside the GEMM.
bool rl_builds(const LinearW& W, const RowTiles& t) { return t.n == 1 && t.R <= 16 && rl_fmt(W) == RL_F16 && (size_t)((W.K + 63) / 64) * t.nt16 * 128 <= 44 * 1024; }

void launch_ln_operands(Model& m, const char* name, const LnOperandsArgs& A) {
    const int threads = (int)round_up((size_t)(A.C / 8), 32);
    // few rows: a CTA per (row, output), each repeating the row statistics; as rows fill the GPU a CTA takes several outputs (more
    // than two CTAs per SM would have to wait for the predecessor's to leave)
    const int gy = std::max(1, std::min(A.nout, 2 * m.num_sms / std::max(A.R, 1)));
    if (threads > kLnMaxThreads) {
        LAUNCH(m, name) {
            launch_pdl(m, ln_operands_wide_kernel, dim3(A.R + A.nseg, gy), dim3(kLnMaxThreads), 0, A);
            check_launch("ln_operands_wide");
        }
        return;
    }
    // Up to 2560 channels there are two variants (ln_operands_kernel says which rows each is for).  The blocks that commit a segment's shift state do not count.
    void (*kernel)(LnOperandsArgs) = ln_operands_kernel<kLnMaxThreads, 1>;
    if (threads <= 320)
        kernel = A.R * gy > ln_resident_blocks(threads) * m.num_sms ? ln_operands_kernel<320, 4> : ln_operands_kernel<320, 3>;
    else if (threads <= 512)
        kernel = ln_operands_kernel<512, 2>;
    LAUNCH(m, name) {
        launch_pdl(m, kernel, dim3(A.R + A.nseg, gy), dim3(threads), 0, A);
        check_launch("ln_operands");
    }
}
// How many chunks of sixteen tokens a step's segments make if they take the matrix form of the WKV (wkv_chunk.cuh says when it is the faster one): all
// of them long, and few enough that the chunk kernel's CTAs have an SM each.  0: token by token.
int wkv_step_chunks(const SegMeta* segs, int nseg, int H, int sms) {
    if (2 * H * nseg > sms) return 0;
    int n = 0;
    for (int i = 0; i < nseg; ++i) {
        if (segs[i].len < kWcMinLen) return 0;
        n += wkv_chunks_of(segs[i].len);
    }
    return n;
}
// Scratch for that many chunks; false where the device has no room for it (the step then goes token by token, which needs none).
bool reserve_wkv_chunks(Model& m, int chunks) {
    return m.ws.wkv_tmp.reserve((size_t)chunks * m.cfg.n_head * kWcFloats * sizeof(float), [&] { RSV_CUDA(cudaStreamSynchronize(m.stream)); });
}
// The raw y of a step in matrix form (wkv7_finish_kernel follows).
void launch_wkv_chunks(int device, cudaStream_t stream, bool pdl, const WkvArgs& A, int chunks) {
    static bool configured[16] = {false};
    if (!configured[device & 15]) {
        RSV_CUDA(cudaFuncSetAttribute(wkv7_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWcSmemAlone));
        configured[device & 15] = true;
    }
    launch_pdl_on(stream, pdl, wkv7_prepare_kernel, dim3(A.H, chunks), dim3(kWcPrepThreads), 0, A);
    launch_pdl_on(stream, pdl, wkv7_chunk_kernel, dim3(2 * A.H, A.nseg), dim3(kWcThreads), kWcSmemAlone, A);
}
int known_parts(int K) { return (K + 8 * kOpThreads - 1) / (8 * kOpThreads); }
void launch_operand_known(Model& m, const float* x, int ldx, int K, const float* amax, int parts, const RowTiles& t, const RlOperandOut& o) {
    LAUNCH(m, "operand_known") {
        launch_pdl(m, operand_known_kernel, dim3(t.R, known_parts(K)), dim3(kOpThreads), 0, x, ldx, K, amax, parts, t.rt, o);
        check_launch("operand_known");
    }
}
void launch_operand_rows(Model& m, const OperandRowsArgs& A) {
    LAUNCH(m, "operand_rows") {
        launch_pdl(m, operand_rows_kernel, dim3((A.R * A.n + kOpThreads / 32 - 1) / (kOpThreads / 32)), dim3(kOpThreads), 0, A);
        check_launch("operand_rows");
    }
}
}  // namespace

void Model::reserve_prompt_scratch(int rows, int segs, int chunk) {
    segs = std::min(segs, num_sms / (2 * std::max(cfg.n_head, 1)));
    rows = (int)std::min<int64_t>(rows, (int64_t)segs * chunk);
    if (segs < 1 || std::min(rows, chunk) < kWcMinLen) return;
    reserve_wkv_chunks(*this, rows / kWcT + segs);  // (every segment may end in a part of a chunk)
}

// ------------------------------------------------------------------------------------------------
// the packed forward step (one token per row), Appendix-style data flow of src/model.rs:396-516
// ------------------------------------------------------------------------------------------------
void Model::forward_rows(State& st, const StepPlan& plan, bool use_cursor) {
    const int R = (int)plan.rows.size(), S = (int)plan.segs.size(), O = (int)plan.out_rows.size();
    const int C = cfg.n_embd, H = cfg.n_head, F = cfg.ffn_hidden, V = cfg.vocab, MIDS = cfg.mids(), NL = cfg.n_layer;
    if (R == 0) return;
    RSV_CUDA(cudaSetDevice(device));
    bool per_group = false, int8 = false;
    for (int i : format_layers)
        for (const LinearW* W : layers[i].big()) {
            per_group = per_group || rl_fmt(*W) == RL_I8G;
            int8 = int8 || rl_fmt(*W) == RL_I8;
        }
    // tw: the layer's launches with many weight tiles; t: the others, which would have too few tiles for the GPU with 128 rows each
    const RowTiles t = row_tiles(R, per_group, true), tw = row_tiles(R, per_group, int8), to = row_tiles(std::max(O, 1), rl_fmt(head) == RL_I8G, rl_fmt(head) == RL_I8);
    // ... cut again where a launch takes several turns of the GPU
    const int fmt = per_group ? RL_I8G : int8 ? RL_I8 : RL_F16, mtc = (C + kRlTileM - 1) / kRlTileM, mtf = (F + kRlTileM - 1) / kRlTileM;
    int mtr = 3 * mtc;
    for (int mid : {cfg.w_mid, cfg.a_mid, cfg.g_mid, cfg.v_mid}) mtr += (mid + kRlTileM - 1) / kRlTileM;
    const int kbc = (C + rl_kelems(fmt) - 1) / rl_kelems(fmt);
    const RowTiles tr = fit_turns(tw, mtr, kbc, fmt, num_sms, R + S), tk = fit_turns(tw, mtf, kbc, fmt, num_sms, R + S), tn = fit_turns(t, mtc, kbc, fmt, num_sms, 0);
    // Operands of a layer, carved again for every layer (a matrix's format is its own); the head's follow the largest layer's.
    OperandCarver cv;
    struct LayerOps {
        RlOperandOut r, w, k, v, a, g, vr, mid[4], y, x2, h;
    };
    auto carve_layer = [&](const LayerW& L, LayerOps& o) {
        cv.used = 0;
        o.r = cv.operand(tr, rl_fmt(L.Wr), C, L.x_r);
        o.k = cv.operand(tr, rl_fmt(L.Wk), C, L.x_k);
        o.v = cv.operand(tr, rl_fmt(L.Wv), C, L.x_v);
        o.w = cv.operand(tr, RL_F16, C, L.x_w);
        o.a = cv.operand(tr, RL_F16, C, L.x_a);
        o.g = cv.operand(tr, RL_F16, C, L.x_g);
        o.vr = rl_fmt(L.Wv) == RL_F16 ? o.v : cv.operand(tr, RL_F16, C, L.x_v);
        const int mids[4] = {cfg.w_mid, cfg.a_mid, cfg.g_mid, cfg.v_mid};
        for (int i = 0; i < 4; ++i) o.mid[i] = cv.operand(t, RL_F16, mids[i]);
        o.y = cv.operand(tn, rl_fmt(L.Wo), C, nullptr, known_parts(C));
        o.x2 = cv.operand(tk, rl_fmt(L.Wfk), C, L.ffn_x_k);
        o.h = cv.operand(tn, rl_fmt(L.Wfv), F, nullptr, known_parts(F));
    };
    LayerOps ops;
    size_t layer_bytes = 0;
    for (int i : format_layers) {
        carve_layer(layers[i], ops);
        layer_bytes = std::max(layer_bytes, cv.used);
    }
    cv.used = layer_bytes;
    RlOperandOut head_op = cv.operand(to, rl_fmt(head), C);
    ensure_operand_memory(*this, cv.used);
    cv.base = ws.op_mem;
    cv.used = layer_bytes;
    head_op = cv.operand(to, rl_fmt(head), C);
    int chunks = plan.multi_row_segments ? wkv_step_chunks(plan.segs.data(), S, H, num_sms) : 0;
    if (chunks && !reserve_wkv_chunks(*this, chunks)) chunks = 0;

    LAUNCH(*this, "embed_ln0") {
        embed_ln0_kernel<<<R, kRowThreads, 0, stream>>>(emb, ln0_w, ln0_b, use_cursor ? ws.tok_list : ws.tokens, use_cursor ? ws.tok_pos : nullptr, R, C, V,
                                                        ws.x, ws.status);
        check_launch("embed_ln0");
    }
    // The residual stream ping-pongs between two buffers: each LayerNorm kernel folds in the pending residual of the
    // linear layer before it (x_cur + pending -> x_alt) so that no linear epilogue has to read-modify-write x.
    float *x_cur = ws.x, *x_alt = ws.x2;
    const float* pending = nullptr;
    const size_t lay_x = (size_t)st.cap * C, lay_s = (size_t)st.cap * H * kHeadSize * kHeadSize;
    // LayerNorm + token shift: commits the shift states staged by the block before (`from` -> `to_state`), stages its own
    auto ln_args = [&](const float* lw, const float* lb, float* shift_state, float* staging, const float* from, float* to_state) {
        LnOperandsArgs A;
        memset(&A, 0, sizeof(A));
        A.x_in = x_cur;
        A.delta = pending;
        A.x_out = pending ? x_alt : nullptr;
        A.lw = lw;
        A.lb = lb;
        A.rows = ws.row_meta;
        A.shift_state = shift_state;
        A.staging = staging;
        A.commit_src = from;
        A.commit_dst = to_state;
        A.segs = ws.seg_meta;
        A.R = R;
        A.C = C;
        A.nseg = from ? S : 0;
        return A;
    };
    float* vgate_buf = ws.xb;
    for (int l = 0; l < NL; ++l) {
        const LayerW& L = layers[l];
        carve_layer(L, ops);
        float* tmix_x = st.tmix_x + l * lay_x;
        float* cmix_x = st.cmix_x + l * lay_x;
        float* wkv = st.wkv + l * lay_s;
        {
            LnOperandsArgs A = ln_args(L.ln1_w, L.ln1_b, tmix_x, ws.staging_t, l ? ws.staging_c : nullptr, l ? cmix_x - lay_x : nullptr);
            const RlOperandOut* out[7] = {&ops.r, &ops.k, &ops.v, &ops.w, &ops.a, &ops.g, &ops.vr};
            const bool shared_v = ops.vr.img == ops.v.img;
            A.nout = l == 0 || shared_v ? 6 : 7;
            A.rt = tr.rt;
            for (int i = 0; i < A.nout; ++i) A.out[i] = *out[i];
            launch_ln_operands(*this, "ln_shift6", A);
        }
        if (pending) {
            std::swap(x_cur, x_alt);
            pending = nullptr;
        }
        float* vgate = l == 0 ? nullptr : vgate_buf;
        {
            // r, k, v and the four rank-space projections in one launch
            float* mw = ws.mid;
            float* ma = mw + cfg.w_mid;
            float* mv = ma + cfg.a_mid;
            float* mg = mv + cfg.v_mid;
            // The rank projections come first: an fp16 row has twice the K blocks of an int8 one, and the last few clusters of the launch find room only when
            // the LayerNorm's CTAs leave (3 rows, 2560 int8 channels: the launch 8.2 -> 6.4 us, a layer 46.6 -> 44.8).
            const RlReq q[7] = {
                {&L.v1, &ops.vr, mv, MIDS, EPI_STORE},  // (layers > 0)
                {&L.w1, &ops.w, mw, MIDS, EPI_TANH},
                {&L.a1, &ops.a, ma, MIDS, EPI_STORE},
                {&L.g1, &ops.g, mg, MIDS, EPI_SIGMOID},
                {&L.Wr, &ops.r, ws.r, C, EPI_STORE},
                {&L.Wk, &ops.k, ws.k, C, EPI_STORE},
                {&L.Wv, &ops.v, ws.v, C, EPI_STORE, nullptr, l == 0 ? ws.vfirst : nullptr},
            };
            run_rows_linear(*this, "linear_rkv_rank", q + (l == 0), 7 - (l == 0), tr);
            // back-projections: decay w, a, gate g and (layers > 0) the v-lerp gate
            const int nb = l == 0 ? 3 : 4;
            const LinearW* Wb[4] = {&L.w2, &L.a2, &L.g2, &L.v2};
            const float* src[4] = {mw, ma, mg, mv};
            bool build = true;
            for (int i = 0; i < nb; ++i) build = build && rl_builds(*Wb[i], t);
            if (!build) {
                OperandRowsArgs A;
                memset(&A, 0, sizeof(A));
                A.R = R;
                A.rt = t.rt;
                A.n = nb;
                for (int i = 0; i < nb; ++i) {
                    A.x[i] = src[i];
                    A.ldx[i] = MIDS;
                    A.K[i] = Wb[i]->K;
                    A.out[i] = ops.mid[i];
                }
                launch_operand_rows(*this, A);
            }
            RlReq q2[4] = {
                {&L.w2, &ops.mid[0], ws.w, C, EPI_DECAY, L.w0},
                {&L.a2, &ops.mid[1], ws.a, C, EPI_SIGMOID_BIAS, L.a0},
                {&L.g2, &ops.mid[2], ws.g, C, EPI_STORE},
                {&L.v2, &ops.mid[3], vgate, C, EPI_SIGMOID_BIAS, L.v0},
            };
            if (build)
                for (int i = 0; i < nb; ++i) {
                    q2[i].op = nullptr;
                    q2[i].x = src[i];
                    q2[i].ldx = MIDS;
                }
            run_rows_linear(*this, "linear_rank_back", q2, nb, t);
        }
        int yparts = H;  // maxima a row of yg comes with
        LAUNCH(*this, "wkv7") {
            const int n_items = H * S;
            if (plan.multi_row_segments) {
                // prefill chunks: vectors built by preparation warps, only state-dependent work in the per-token chain (wkv_seq.cuh)
                // few (head, segment) pairs: a head over two CTAs
                if (chunks > 0) {
                    launch_wkv_chunks(device, stream, use_pdl, WkvArgs{ws.seg_meta, ws.r, ws.k, ws.v, vgate, ws.vfirst, ws.w, ws.a, L.k_k, L.k_a, wkv, l == 0 ? st.v_first : nullptr, ws.yg, ws.wkv_tmp.as<float>(), S, H, C, ws.status}, chunks);
                } else if (H * S <= num_sms) {
                    // Where every CTA can have an SM to itself it asks for more than half of the shared memory, so that no two share one:
                    // they would start in pairs as the predecessor's CTAs leave, and a pair takes a third longer (512 tokens, 40 heads).
                    const size_t alone = 2 * H * S <= num_sms ? 120 * 1024 : 0;
                    static bool configured[16] = {false};
                    if (!configured[device & 15]) {
                        RSV_CUDA(cudaFuncSetAttribute(wkv7_seq_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024));
                        configured[device & 15] = true;
                    }
                    launch_pdl(*this, wkv7_seq_kernel<2>, dim3(2 * H, S), dim3(kWsThreads), alone, ws.seg_meta, ws.r, ws.k, ws.v, vgate, ws.vfirst, ws.w, ws.a, ws.g,
                               L.k_k, L.k_a, L.r_k, L.lnx_w, L.lnx_b, wkv, l == 0 ? st.v_first : nullptr, ws.yg, H, C, ws.status);
                } else {
                    launch_pdl(*this, wkv7_seq_kernel<4>, dim3(H, S), dim3(kWsThreads), 0, ws.seg_meta, ws.r, ws.k, ws.v, vgate, ws.vfirst, ws.w, ws.a, ws.g,
                               L.k_k, L.k_a, L.r_k, L.lnx_w, L.lnx_b, wkv, l == 0 ? st.v_first : nullptr, ws.yg, H, C, ws.status);
                }
                launch_pdl(*this, wkv7_finish_kernel, dim3((R * H + kWsFinishThreads / 32 - 1) / (kWsFinishThreads / 32)), dim3(kWsFinishThreads), 0, ws.r, ws.k,
                           ws.v, vgate, ws.vfirst, ws.a, ws.g, L.k_a, L.r_k, L.lnx_w, L.lnx_b, ws.yg, R, H, C, ws.ymax);
            } else if (wr_pays(n_items, num_sms)) {
                // many (session, head) pairs: one state row per lane, states staged by TMA (wkv_rows.cuh)
                const size_t rows_total = (size_t)cfg.n_layer * st.cap * H * kHeadSize;
                if (rows_total >= (1ull << 31)) throw std::runtime_error("state too large for the 32-bit row coordinate of its tensor map");
                if (!st.wkv_map_ok) {
                    encode_state_map(&st.wkv_map, st.wkv, rows_total);
                    st.wkv_map_ok = true;
                }
                static bool configured[16] = {false};
                if (!configured[device & 15]) {
                    RSV_CUDA(cudaFuncSetAttribute(wkv7_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWrSmemBytes));
                    configured[device & 15] = true;
                }
                if (C % 64) throw std::runtime_error("n_embd must be a multiple of 64");
                const int ctas = std::min((n_items + kWrPairs - 1) / kWrPairs, num_sms);
                launch_pdl(*this, wkv7_rows_kernel, dim3(ctas), dim3(kWrThreads), kWrSmemBytes, st.wkv_map, (long long)l * st.cap * H * kHeadSize, ws.seg_meta,
                           n_items, ws.r, ws.k, ws.v, vgate, ws.vfirst, ws.w, ws.a, ws.g, L.k_k, L.k_a, L.r_k, L.lnx_w, L.lnx_b,
                           l == 0 ? st.v_first : nullptr, ws.yg, H, C, ws.status, ws.ymax);
                yparts = 2 * H;
            } else {
                launch_pdl(*this, wkv7_kernel, dim3(H, S), dim3(kWkvThreads), 0, ws.seg_meta, ws.r, ws.k, ws.v, vgate, ws.vfirst, ws.w, ws.a, ws.g, L.k_k, L.k_a,
                           L.r_k, L.lnx_w, L.lnx_b, wkv, l == 0 ? st.v_first : nullptr, ws.yg, H, C, ws.ymax);
            }
            check_launch("wkv7");
        }
        // a linear layer on activations whose row maxima their producer collected
        auto linear_known = [&](const char* name, RlReq q, const float* x, int ldx, const float* amax, int parts, const RlOperandOut& op) {
            launch_operand_known(*this, x, ldx, q.W->K, amax, parts, tn, op);
            q.op = &op;
            run_rows_linear(*this, name, &q, 1, tn);
        };
        linear_known("linear_att_out", RlReq{&L.Wo, nullptr, ws.delta, C, EPI_STORE}, ws.yg, C, ws.ymax, yparts, ops.y);
        pending = ws.delta;
        {
            LnOperandsArgs A = ln_args(L.ln2_w, L.ln2_b, cmix_x, ws.staging_c, ws.staging_t, tmix_x);
            A.rt = tk.rt;
            A.nout = 1;
            A.out[0] = ops.x2;
            launch_ln_operands(*this, "ln_shift1", A);
        }
        std::swap(x_cur, x_alt);
        pending = nullptr;
        {
            RlReq q = {&L.Wfk, &ops.x2, ws.h, F, EPI_RELU2};
            q.ymax = ws.hmax;
            run_rows_linear(*this, "linear_ffn_key", &q, 1, tk);
        }
        linear_known("linear_ffn_value", RlReq{&L.Wfv, nullptr, ws.delta, C, EPI_STORE}, ws.h, F, ws.hmax, (F + kRlTileM - 1) / kRlTileM, ops.h);
        pending = ws.delta;
    }
    LAUNCH(*this, "commit_shift") {
        launch_pdl(*this, commit_shift_kernel, dim3(S), dim3(256), 0, ws.staging_c, ws.seg_meta, C, st.cmix_x + (size_t)(NL - 1) * lay_x);
        check_launch("commit_shift");
    }
    ws.final_x = x_cur;
    ws.final_delta = pending;
    if (O) {
        LnOperandsArgs A;
        memset(&A, 0, sizeof(A));
        A.x_in = x_cur;
        A.delta = pending;
        A.lw = ln_out_w;
        A.lb = ln_out_b;
        A.row_map = ws.out_rows;
        A.R = O;
        A.C = C;
        A.rt = to.rt;
        A.nout = 1;
        A.out[0] = head_op;
        launch_ln_operands(*this, "ln_out", A);
        RlReq q = {&head, &head_op, ws.logits, V, EPI_STORE};
        run_rows_linear(*this, "linear_head", &q, 1, to);
    }
    if (use_cursor) LAUNCH(*this, "advance_cursor") {
            advance_cursor_kernel<<<1, 1, 0, stream>>>(ws.tok_pos);
            check_launch("advance_cursor");
        }
}


// ------------------------------------------------------------------------------------------------
// batch-1 weight-streaming decode kernel: host side
// ------------------------------------------------------------------------------------------------
namespace {

template <int CMAX>
void launch_stream(const DsParams& P, int grid, size_t smem, cudaStream_t stream, bool configure_only) {
    if (configure_only) {
        RSV_CUDA(cudaFuncSetAttribute(decode_stream_kernel<CMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        // the consumers' larger register share (setmaxnreg) exists only if the block was launched with this much
        cudaFuncAttributes fa;
        RSV_CUDA(cudaFuncGetAttributes(&fa, decode_stream_kernel<CMAX>));
        if (fa.numRegs < kDsLaunchRegs) throw std::runtime_error("weight-streaming decode kernel: built with too few registers");
        RSV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_stream_kernel<CMAX>, kDsThreads, smem));
        if (per_sm < 1) throw std::runtime_error("weight-streaming decode kernel does not fit on an SM");
        return;
    }
    void* args[] = {(void*)&P};
    RSV_CUDA(cudaLaunchCooperativeKernel((const void*)decode_stream_kernel<CMAX>, dim3(grid), dim3(kDsThreads), args, smem, stream));
}
void dispatch_stream(int cmax, const DsParams& P, int grid, size_t smem, cudaStream_t stream, bool configure_only) {
    switch (cmax) {
        case 512: return launch_stream<512>(P, grid, smem, stream, configure_only);
        case 1024: return launch_stream<1024>(P, grid, smem, stream, configure_only);
        case 2048: return launch_stream<2048>(P, grid, smem, stream, configure_only);
        case 2560: return launch_stream<2560>(P, grid, smem, stream, configure_only);
        case 4096: return launch_stream<4096>(P, grid, smem, stream, configure_only);
        default: throw std::runtime_error("weight-streaming decode kernel: unsupported n_embd");
    }
}

}  // namespace

bool Model::stream_available() {
    if (!use_stream) return false;
    StreamCtx& sc = sctx;
    if (sc.tried) return sc.ok;
    sc.tried = true;
    auto fail = [&](const std::string& why) {
        sc.why = why;
        sc.ok = false;
        if (const char* e = getenv("RSV_VERBOSE"))
            if (*e && *e != '0') fprintf(stderr, "[rsv] weight-streaming decode kernel not used: %s\n", why.c_str());
        return false;
    };
    RSV_CUDA(cudaSetDevice(device));
    int coop = 0;
    RSV_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    if (!coop) return fail("device does not support cooperative launches");
    const int L = cfg.n_layer, C = cfg.n_embd, F = cfg.ffn_hidden, V = cfg.vocab, H = cfg.n_head, G = num_sms;
    // int8 matrices: one (scale, zero) per output row, or the reference container's one per row and group of 128 weights
    auto format_of = [](const LinearW& W) { return W.wtype != W_INT8 ? 0 : (W.wscale && W.wzero) ? 1 : W.sz ? 2 : -1; };
    if (format_of(head) < 0) return fail("int8 head without scales");
    const int fmt = layers.empty() ? 0 : format_of(layers[0].Wr);
    for (const LayerW& Lw : layers)
        for (const LinearW* W : Lw.big())
            if (format_of(*W) != fmt || fmt < 0) return fail("the big matrices of the layers differ in their weight format, or an int8 matrix has no scales");
    // the layout (row ownership, chunks, shared memory, every capacity of the kernel's tables) is pure arithmetic on the shape
    const DsShape shp{L, C, F, V, H, cfg.w_mid, cfg.a_mid, cfg.v_mid, cfg.g_mid, fmt, format_of(head)};
    DsLayout lay;
    {
        std::string why;
        if (!ds_layout(shp, G, lay, why)) return fail(why);
    }
    const int cmax = lay.cmax, vec_floats = lay.vec_floats, ring_bytes = lay.ring_bytes;
    sc.kl = cmax;
    sc.grid = G;
    sc.ring_bytes = ring_bytes;
    sc.vec_floats = vec_floats;
    sc.smem = lay.smem;
    DsParams P;
    memset(&P, 0, sizeof(P));
    try {
        dispatch_stream(cmax, P, G, sc.smem, stream, true);
    } catch (const std::exception& e) {
        return fail(e.what());
    }
    // per-layer tables: sizes and CTA groups from the layout, pointers from the checkpoint
    auto bind = [&](DsEntry& e, const LinearW& W, const float* mix) -> bool {
        if (e.M != 0 && (W.M != e.M || (e.is_i8 ? W.K : 2 * W.K) != e.row_stride)) return false;
        e.base = (const char*)W.w;
        e.wscale = W.wscale;
        e.wzero = W.wzero;
        e.sz = W.sz;
        e.mix = mix;
        return true;
    };
    std::vector<DsLayer> dl((size_t)L);
    for (int l = 0; l < L; ++l) {
        const LayerW& Lw = layers[l];
        DsLayer& d = dl[l];
        memset(&d, 0, sizeof(d));
        ds_layer_entries(shp, G, l > 0, d.e);
        if (!(bind(d.e[DSE_W1], Lw.w1, Lw.x_w) && bind(d.e[DSE_A1], Lw.a1, Lw.x_a) && bind(d.e[DSE_G1], Lw.g1, Lw.x_g) && bind(d.e[DSE_V1], Lw.v1, Lw.x_v) &&
              bind(d.e[DSE_WR], Lw.Wr, Lw.x_r) && bind(d.e[DSE_WK], Lw.Wk, Lw.x_k) && bind(d.e[DSE_WV], Lw.Wv, Lw.x_v) && bind(d.e[DSE_WO], Lw.Wo, nullptr) &&
              bind(d.e[DSE_WFK], Lw.Wfk, nullptr) && bind(d.e[DSE_WFV], Lw.Wfv, nullptr)))
            return fail("a matrix of the checkpoint does not have the model's shape");
        for (const LinearW* W : {&Lw.w1, &Lw.a1, &Lw.g1, &Lw.v1})
            if (W->wtype != W_F16) return fail("rank projections must be fp16 [mid, n_embd]");
        d.w2 = (const __half*)Lw.w2.w;
        d.a2 = (const __half*)Lw.a2.w;
        d.v2 = (const __half*)Lw.v2.w;
        d.g2 = (const __half*)Lw.g2.w;
        d.ln1_w = Lw.ln1_w;
        d.ln1_b = Lw.ln1_b;
        d.ln2_w = Lw.ln2_w;
        d.ln2_b = Lw.ln2_b;
        d.lnx_w = Lw.lnx_w;
        d.lnx_b = Lw.lnx_b;
        d.x_r = Lw.x_r;
        d.x_k = Lw.x_k;
        d.x_v = Lw.x_v;
        d.ffn_x_k = Lw.ffn_x_k;
        d.w0 = Lw.w0;
        d.a0 = Lw.a0;
        d.v0 = Lw.v0;
        d.r_k = Lw.r_k;
        d.k_k = Lw.k_k;
        d.k_a = Lw.k_a;
    }
    RSV_CUDA(device_malloc(&sc.d_layers, dl.size() * sizeof(DsLayer)));
    RSV_CUDA(cudaMemcpy(sc.d_layers, dl.data(), dl.size() * sizeof(DsLayer), cudaMemcpyHostToDevice));
    {
        // second copy of the weights in the order the kernel consumes them (a chunk = one bulk copy): region sizes = the largest CTA's
        const long long wslot = lay.wslot, hslot = lay.hslot;
        DsEntry head_e = ds_head_entry(shp, G);
        if (!bind(head_e, head, nullptr)) return fail("the head of the checkpoint does not have the model's shape");
        sc.wslot = wslot;
        sc.hslot = hslot;
        RSV_CUDA(device_malloc(&sc.wstream, (size_t)wslot * G * L));
        RSV_CUDA(device_malloc(&sc.hstream, (size_t)hslot * G));
        DsParams Q;
        memset(&Q, 0, sizeof(Q));
        Q.layers = (const DsLayer*)sc.d_layers;
        Q.head = head_e;
        Q.L = L;
        Q.H = H;
        Q.wm = cfg.w_mid;
        Q.am = cfg.a_mid;
        Q.vm = cfg.v_mid;
        Q.gm = cfg.g_mid;
        ds_retile_kernel<<<G, 256, 0, stream>>>(Q, (char*)sc.wstream, wslot, (char*)sc.hstream, hslot);
        check_launch("ds_retile");
        RSV_CUDA(cudaStreamSynchronize(stream));
        if (const char* e = getenv("RSV_VERBOSE"))
            if (*e && *e != '0')
                fprintf(stderr, "[rsv] weight-streaming decode kernel: %.2f GB second copy of the weights in consumption order (%lld bytes per layer and SM); ring %d bytes%s\n",
                        ((double)wslot * G * L + (double)hslot * G) / 1e9, wslot, ring_bytes, lay.head_early ? ", a head's first chunk released early" : "");
    }
    const size_t pairs = (size_t)7 * C + cfg.mids();
    sc.exchange_bytes = pairs * 8 + (size_t)F * 4;
    RSV_CUDA(device_malloc(&sc.exchange, sc.exchange_bytes));
    RSV_CUDA(cudaMemsetAsync(sc.exchange, 0, sc.exchange_bytes, stream));  // tag 0: no launch's
    RSV_CUDA(device_malloc(&sc.cand_val, (size_t)G * 4));
    RSV_CUDA(device_malloc(&sc.cand_idx, (size_t)G * 4));
    RSV_CUDA(device_malloc(&sc.grid_bar, 4));
    RSV_CUDA(cudaMemsetAsync(sc.grid_bar, 0, 4, stream));
    P.layers = (const DsLayer*)sc.d_layers;
    P.head = ds_head_entry(shp, G);
    bind(P.head, head, nullptr);
    P.emb = emb;
    P.ln0_w = ln0_w;
    P.ln0_b = ln0_b;
    P.lno_w = ln_out_w;
    P.lno_b = ln_out_b;
    P.L = L;
    P.C = C;
    P.H = H;
    P.F = F;
    P.V = V;
    P.wm = cfg.w_mid;
    P.am = cfg.a_mid;
    P.vm = cfg.v_mid;
    P.gm = cfg.g_mid;
    P.xa = sc.exchange;
    P.xb = P.xa + C;
    P.yg = P.xb + C;
    P.vfirst = P.yg + C;
    P.rkv = P.vfirst + C;
    P.mid = P.rkv + 3 * (size_t)C;
    P.hbuf = (uint32_t*)(P.mid + cfg.mids());
    P.cand_val = sc.cand_val;
    P.cand_idx = sc.cand_idx;
    P.grid_bar = sc.grid_bar;
    P.wstream = (const char*)sc.wstream;
    P.wslot = sc.wslot;
    P.hstream = (const char*)sc.hstream;
    P.hslot = sc.hslot;
    P.ring_bytes = ring_bytes;
    P.vec_floats = vec_floats;
    sc.params_template.resize(sizeof(DsParams));
    memcpy(sc.params_template.data(), &P, sizeof(P));
    sc.ok = true;
    return true;
}

void Model::run_stream(State& st, int slot, int n_tokens, bool tok_from_list, bool argmax_feed, uint32_t* seq_dev, int* seq_cnt_dev, int seq_cap,
                       const uint32_t* host_token) {
    if (!stream_available()) throw std::runtime_error("weight-streaming decode path unavailable: " + sctx.why);
    StreamCtx& sc = sctx;
    RSV_CUDA(cudaSetDevice(device));
    if (slot < 0 || slot >= st.cap) throw std::runtime_error("state slot out of range");
    ensure_workspace(1, 1, 1);
    DsParams P;
    memcpy(&P, sc.params_template.data(), sizeof(P));
    P.slot = slot;
    P.lay_x = (long long)st.cap * cfg.n_embd;
    P.lay_s = (long long)st.cap * cfg.n_head * kHeadSize * kHeadSize;
    P.tmix_x = st.tmix_x;
    P.wkv = st.wkv;
    P.cmix_x = st.cmix_x;
    P.state_vfirst = st.v_first;
    P.tokens = ws.tokens;
    P.tok_list = ws.tok_list;
    P.seq = seq_dev;
    P.seq_cnt = seq_cnt_dev;
    P.seq_cap = seq_cap;
    P.logits = ws.logits;
    P.status = ws.status;
    P.n_tokens = n_tokens;
    P.tok_from_list = host_token ? 2 : tok_from_list ? 1 : 0;
    P.tok0 = host_token ? *host_token : 0u;
    P.argmax_feed = argmax_feed ? 1 : 0;
    sc.seq.run((uint32_t)n_tokens * (uint32_t)cfg.n_layer, (unsigned)sc.grid * (unsigned)(argmax_feed ? n_tokens : n_tokens - 1), [&](uint32_t epoch, unsigned bar_base) {
        P.epoch = epoch;
        P.bar_base = bar_base;
        LAUNCH(*this, "decode_stream") { dispatch_stream(sc.kl, P, sc.grid, sc.smem, stream, false); }
    });
}

void Model::check_status() {
    int sw[2] = {0, 0};  // status bits; where the weight-streaming decode kernel gave up
    RSV_CUDA(cudaMemcpyAsync(sw, ws.status, 2 * sizeof(int), cudaMemcpyDeviceToHost, stream));
    RSV_CUDA(cudaStreamSynchronize(stream));
    judge_status(sw);
}

void Model::judge_status(const int* sw) {
    const int s = sw[0];
    if (s) {
        RSV_CUDA(cudaMemsetAsync(ws.status, 0, 2 * sizeof(int), stream));
        if ((s & 32) && sctx.exchange) {  // a launch that gave up left some of its exchanged values unwritten
            RSV_CUDA(cudaMemsetAsync(sctx.exchange, 0, sctx.exchange_bytes, stream));
            RSV_CUDA(cudaMemsetAsync(sctx.grid_bar, 0, 4, stream));
            sctx.seq = StreamSequence{};
        }
        if (s & 32) {
            static const char* const site[5] = {"a wait", "a chunk of weight rows", "room in the ring", "a grid barrier", "a chunk of a head's rows"};
            const int k = sw[1] & 15;
            throw std::runtime_error(std::string("weight-streaming decode kernel gave up waiting for ") + site[k >= 1 && k <= 4 ? k : 0] + " (device status bit 5; CTA " +
                                     std::to_string((sw[1] >> 20) & 255) + ", index " + std::to_string((sw[1] >> 4) & 0xFFFF) + ")");
        }
        if (s & 16) throw std::runtime_error("WKV kernel gave up waiting for a staged state (device status bit 4)");
        if (s & 8) throw std::runtime_error("weight-streaming decode kernel: chunk table too small for this shape (device status bit 3)");
        if (s & 2) throw std::runtime_error("tensor-core kernel gave up waiting on a barrier (device status bit 1)");
        if (s & 1) throw std::runtime_error("token id out of range (>= vocab); the embedding row 0 was used instead");
        throw std::runtime_error("device status word = " + std::to_string(s));
    }
}

// ------------------------------------------------------------------------------------------------
// helpers used by the C ABI
// ------------------------------------------------------------------------------------------------
void engine_argmax(Model& m, const float* logits_dev, int rows, uint32_t* next_tok_dev, uint32_t* seq_dev, int* seq_cnt_dev, int seq_cap,
                   const int* row_map_dev) {
    LAUNCH(m, "argmax") {
        argmax_rows_kernel<<<rows, kArgmaxThreads, 0, m.stream>>>(logits_dev, m.cfg.vocab, next_tok_dev, seq_dev, seq_cnt_dev, seq_cap, row_map_dev);
        check_launch("argmax");
    }
}

// Up to 65536 logits (eight CTAs, the portable cluster size, of 8192) a row is a cluster of CTAs that hold it in registers: 25 us for
// 65536 logits with top-k 50 + top-p against 218 us; larger vocabularies go through the one-CTA kernel and its work area.
static void launch_sample(cudaStream_t stream, const float* logits_dev, int rows, int V, const float* sampler8_dev, const uint32_t* hist_dev, int hist_stride,
                          const int* round_cnt_dev, float* temp_dev, uint32_t* counter_dev, uint32_t* next_tok_dev, uint32_t* seq_dev, int* seq_cnt_dev,
                          int seq_cap, const int* row_map_dev) {
    if (V <= kScMaxV) {
        const int S = (V + kScSeg - 1) / kScSeg;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)rows * S);
        cfg.blockDim = dim3(kScThreads);
        cfg.dynamicSmemBytes = hist_dev ? kScSeg * sizeof(uint32_t) : 0;
        cfg.stream = stream;
        cudaLaunchAttribute at[1];
        memset(at, 0, sizeof(at));
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)S;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        RSV_CUDA(cudaLaunchKernelEx(&cfg, sample_cluster_kernel, logits_dev, V, sampler8_dev, hist_dev, hist_stride, round_cnt_dev, next_tok_dev, seq_dev, seq_cnt_dev,
                                    seq_cap, row_map_dev, S));
    } else {
        sample_rows_kernel<<<rows, kSampleThreads, 0, stream>>>(logits_dev, V, sampler8_dev, hist_dev, hist_stride, round_cnt_dev, temp_dev, counter_dev, next_tok_dev,
                                                                seq_dev, seq_cnt_dev, seq_cap, row_map_dev);
    }
    check_launch("sample");
}

void engine_sample(Model& m, const float* logits_dev, int rows, const float* sampler8_dev, const uint32_t* hist_dev, int hist_stride,
                   const int* round_cnt_dev, uint32_t* next_tok_dev, uint32_t* seq_dev, int* seq_cnt_dev, int seq_cap, const int* row_map_dev) {
    if (rows > m.ws.outs) throw std::runtime_error("engine_sample: more rows than the work area holds");
    LAUNCH(m, "sample") {
        launch_sample(m.stream, logits_dev, rows, m.cfg.vocab, sampler8_dev, hist_dev, hist_stride, round_cnt_dev, m.ws.samp_temp, m.ws.samp_cnt, next_tok_dev, seq_dev,
                      seq_cnt_dev, seq_cap, row_map_dev);
    }
}

void engine_sample_raw(cudaStream_t stream, const float* logits_dev, int rows, int V, const float* sampler8_dev, const uint32_t* hist_dev,
                       int hist_stride, float* temp_dev, uint32_t* counter_dev, uint32_t* out_dev) {
    launch_sample(stream, logits_dev, rows, V, sampler8_dev, hist_dev, hist_stride, nullptr, temp_dev, counter_dev, out_dev, nullptr, nullptr, 0, nullptr);
}

Ticket::~Ticket() {
    if (model) {
        cudaSetDevice(model->device);
        if (graph_exec || graph) cudaStreamSynchronize(model->stream);
    }
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    if (graph) cudaGraphDestroy(graph);
    if (seq) cudaFree(seq);
    if (cnt) cudaFree(cnt);
    if (sampler) cudaFree(sampler);
}

void engine_merge_tokens(Model& m, const uint32_t* host_tok_dev, const uint32_t* slot_tok_dev, int R) {
    LAUNCH(m, "merge_tokens") {
        merge_tokens_kernel<<<(R + 255) / 256, 256, 0, m.stream>>>(host_tok_dev, m.ws.row_meta, slot_tok_dev, R, m.ws.tokens);
        check_launch("merge_tokens");
    }
}

void engine_argmax_raw(cudaStream_t stream, const float* logits_dev, int rows, int V, uint32_t* out_dev) {
    argmax_rows_kernel<<<rows, kArgmaxThreads, 0, stream>>>(logits_dev, V, out_dev, nullptr, nullptr, 0, nullptr);
    check_launch("argmax");
}

void engine_dequant_int8(cudaStream_t stream, const uint8_t* idx_dev, const uint32_t* sz_dev, size_t M, size_t K, float* out_dev) {
    dequant_int8_kernel<<<148 * 8, 256, 0, stream>>>(idx_dev, sz_dev, M, K, out_dev);
    check_launch("dequant_int8");
}


void engine_quantize_int8(cudaStream_t stream, const float* w_dev, size_t M, size_t K, uint8_t* idx_dev, uint32_t* sz_dev) {
    const size_t groups = M * (K / 128);
    const int blocks = (int)std::min<size_t>((groups + 7) / 8, 148 * 16);
    quantize_int8_kernel<<<blocks, 256, 0, stream>>>(w_dev, groups, idx_dev, sz_dev);
    check_launch("quantize_int8");
}

void engine_segment_sums(Model& m, int n_segments, float* acc_dev) {
    if (!m.ws.final_x) throw std::runtime_error("segment sums: no step has run");
    LAUNCH(m, "segment_sums") {
        segment_sums_kernel<<<dim3(n_segments, (m.cfg.n_embd + 255) / 256), 256, 0, m.stream>>>(m.ws.final_x, m.ws.final_delta, m.ws.seg_meta, m.cfg.n_embd, acc_dev);
        check_launch("segment_sums");
    }
}

// Operator-level WKV-7 step on host data (see the declaration).  The four kernels are launched as forward_rows launches them.
void engine_op_wkv7(int device, int variant, int nseg, int T, int H, const float* const in[8], const float* const par[5], float* state_host, float* y_host) {
    RSV_CUDA(cudaSetDevice(device));
    const int C = H * kHeadSize, R = nseg * T;
    const size_t row_bytes = (size_t)R * C * 4, st_floats = (size_t)nseg * H * kHeadSize * kHeadSize;
    struct Buf {
        void* p = nullptr;
        ~Buf() {
            if (p) cudaFree(p);
        }
    };
    Buf din[8], dpar[5], dstate, dy, dseg, dstatus, dtmp;
    for (int i = 0; i < 8; ++i)
        if (in[i]) {
            RSV_CUDA(device_malloc(&din[i].p, row_bytes));
            RSV_CUDA(cudaMemcpy(din[i].p, in[i], row_bytes, cudaMemcpyHostToDevice));
        }
    for (int i = 0; i < 5; ++i) {
        RSV_CUDA(device_malloc(&dpar[i].p, (size_t)C * 4));
        RSV_CUDA(cudaMemcpy(dpar[i].p, par[i], (size_t)C * 4, cudaMemcpyHostToDevice));
    }
    RSV_CUDA(device_malloc(&dstate.p, st_floats * 4));
    RSV_CUDA(cudaMemcpy(dstate.p, state_host, st_floats * 4, cudaMemcpyHostToDevice));
    RSV_CUDA(device_malloc(&dy.p, row_bytes));
    RSV_CUDA(cudaMemset(dy.p, 0, row_bytes));
    std::vector<SegMeta> segs((size_t)nseg);
    for (int s2 = 0; s2 < nseg; ++s2) segs[s2] = SegMeta{s2 * T, T, s2, 0};
    RSV_CUDA(device_malloc(&dseg.p, segs.size() * sizeof(SegMeta)));
    RSV_CUDA(cudaMemcpy(dseg.p, segs.data(), segs.size() * sizeof(SegMeta), cudaMemcpyHostToDevice));
    RSV_CUDA(device_malloc(&dstatus.p, 8));
    RSV_CUDA(cudaMemset(dstatus.p, 0, 8));
    const float *r = (const float*)din[0].p, *k = (const float*)din[1].p, *v = (const float*)din[2].p, *w = (const float*)din[3].p, *a = (const float*)din[4].p,
                *g = (const float*)din[5].p, *vgate = (const float*)din[6].p, *vfirst = (const float*)din[7].p;
    const float *k_k = (const float*)dpar[0].p, *k_a = (const float*)dpar[1].p, *r_k = (const float*)dpar[2].p, *lnx_w = (const float*)dpar[3].p,
                *lnx_b = (const float*)dpar[4].p;
    float *state = (float*)dstate.p, *yg = (float*)dy.p;
    int* status = (int*)dstatus.p;
    const SegMeta* sm = (const SegMeta*)dseg.p;
    cudaDeviceProp prop;
    RSV_CUDA(cudaGetDeviceProperties(&prop, device));
    const int sms = prop.multiProcessorCount, n_items = H * nseg;
    if (variant < 0 || variant > 4) throw std::runtime_error("wkv7: variant must be 0 (automatic), 1 (token kernel), 2 (row-per-lane kernel), 3 or 4 (sequence kernel, head over two CTAs / one CTA)");
    // automatic: what a step runs.  A step's decays are exp(-sigmoid / sqrt(e)) > 0.54; products of sixteen others (which only this entry point can be given)
    // may underflow: those go token by token.
    constexpr int kChunked = 5;
    int chunks = 0;
    if (variant == 0) {
        chunks = T > 1 ? wkv_step_chunks(segs.data(), nseg, H, sms) : 0;
        for (size_t i = 0; i < (size_t)R * C && chunks; ++i)
            if (!(in[3][i] >= 0.5f && in[3][i] <= 1.0f)) chunks = 0;
        if (chunks && device_malloc(&dtmp.p, (size_t)chunks * H * kWcFloats * sizeof(float)) != cudaSuccess) {
            dtmp.p = nullptr;
            cudaGetLastError();
            chunks = 0;
        }
        variant = chunks ? kChunked : T > 1 ? (n_items <= sms ? 3 : 4) : (n_items >= 4 * sms ? 2 : 1);
    }
    if (variant == 1) {
        wkv7_kernel<<<dim3(H, nseg), kWkvThreads>>>(sm, r, k, v, vgate, vfirst, w, a, g, k_k, k_a, r_k, lnx_w, lnx_b, state, nullptr, yg, H, C, nullptr);
    } else if (variant == 2) {
        CUtensorMap map;
        encode_state_map(&map, state, (size_t)nseg * H * kHeadSize);
        RSV_CUDA(cudaFuncSetAttribute(wkv7_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWrSmemBytes));
        const int ctas = std::min((n_items + kWrPairs - 1) / kWrPairs, sms);
        wkv7_rows_kernel<<<ctas, kWrThreads, kWrSmemBytes>>>(map, 0LL, sm, n_items, r, k, v, vgate, vfirst, w, a, g, k_k, k_a, r_k, lnx_w, lnx_b, nullptr, yg, H, C, status, nullptr);
    } else {
        if (variant == kChunked) {
            for (int s2 = 0, before = 0; s2 < nseg; before += wkv_chunks_of(T), ++s2) segs[s2].chunk0 = before;
            RSV_CUDA(cudaMemcpy(dseg.p, segs.data(), segs.size() * sizeof(SegMeta), cudaMemcpyHostToDevice));
            launch_wkv_chunks(device, nullptr, false, WkvArgs{sm, r, k, v, vgate, vfirst, w, a, k_k, k_a, state, nullptr, yg, (float*)dtmp.p, nseg, H, C, status}, chunks);
        } else if (variant == 3)
            wkv7_seq_kernel<2><<<dim3(2 * H, nseg), kWsThreads>>>(sm, r, k, v, vgate, vfirst, w, a, g, k_k, k_a, r_k, lnx_w, lnx_b, state, nullptr, yg, H, C, status);
        else
            wkv7_seq_kernel<4><<<dim3(H, nseg), kWsThreads>>>(sm, r, k, v, vgate, vfirst, w, a, g, k_k, k_a, r_k, lnx_w, lnx_b, state, nullptr, yg, H, C, status);
        check_launch("wkv7_seq");
        wkv7_finish_kernel<<<(R * H + kWsFinishThreads / 32 - 1) / (kWsFinishThreads / 32), kWsFinishThreads>>>(r, k, v, vgate, vfirst, a, g, k_a, r_k, lnx_w, lnx_b, yg,
                                                                                                              R, H, C, nullptr);
    }
    check_launch("wkv7");
    RSV_CUDA(cudaDeviceSynchronize());
    int st = 0;
    RSV_CUDA(cudaMemcpy(&st, status, 4, cudaMemcpyDeviceToHost));
    if (st) throw std::runtime_error("WKV kernel gave up waiting for a staged state (device status " + std::to_string(st) + ")");
    RSV_CUDA(cudaMemcpy(state_host, state, st_floats * 4, cudaMemcpyDeviceToHost));
    RSV_CUDA(cudaMemcpy(y_host, yg, row_bytes, cudaMemcpyDeviceToHost));
}

void engine_op_linear(Model& m, int path, int wtype, const void* w_host, const uint32_t* sz_host, int M, int K, const float* x_host, int R,
                      float* y_host) {
    RSV_CUDA(cudaSetDevice(m.device));
    if (M < 1 || K < 8 || R < 1) throw std::runtime_error("op_linear: empty problem");
    if (wtype == W_INT8 ? (K % 128 != 0) : (K % 8 != 0)) throw std::runtime_error("op_linear: K must be a multiple of 128 (int8) or 8 (fp16)");
    Loader ld{m, nullptr};
    LinearW W;
    W.M = M;
    W.K = K;
    W.wtype = wtype;
    const size_t first_alloc = m.allocs.size();
    float *dx = nullptr, *dy = nullptr;
    try {
        if (wtype == W_INT8) {
            W.w = ld.upload(w_host, (size_t)M * K);
            W.sz = (uint32_t*)ld.upload(sz_host, (size_t)M * (K / 128) * 4);
            ld.prepare_tc_i8(W, sz_host);
        } else {
            W.w = ld.upload(w_host, (size_t)M * K * 2);
            ld.prepare_tc_f16(W);
        }
        if (path == 1 && wtype == W_INT8 && (!W.row_scaled() || M % kTcTileM)) throw std::runtime_error("op_linear: this matrix cannot take the tensor-core path (needs one scale/zero per row, M and K multiples of 128)");
        RSV_CUDA(device_malloc(&dx, (size_t)R * K * 4));
        RSV_CUDA(device_malloc(&dy, (size_t)R * M * 4));
        RSV_CUDA(cudaMemcpyAsync(dx, x_host, (size_t)R * K * 4, cudaMemcpyHostToDevice, m.stream));
        if (path == 1) {
            const RowTiles t = row_tiles(R, false, rl_fmt(W) == RL_I8);
            OperandCarver cv;
            cv.operand(t, rl_fmt(W), K);
            ensure_operand_memory(m, cv.used);
            cv.base = m.ws.op_mem;
            cv.used = 0;
            OperandRowsArgs A;
            memset(&A, 0, sizeof(A));
            A.R = R;
            A.rt = t.rt;
            A.n = 1;
            A.x[0] = dx;
            A.ldx[0] = A.K[0] = K;
            A.out[0] = cv.operand(t, rl_fmt(W), K);
            launch_operand_rows(m, A);
            RlReq q = {&W, &A.out[0], dy, M, EPI_STORE};
            run_rows_linear(m, "op_linear", &q, 1, t);
        } else {
            run_linear_simt(m, "op_linear_simt", W, dx, dy, R);
        }
        RSV_CUDA(cudaMemcpyAsync(y_host, dy, (size_t)R * M * 4, cudaMemcpyDeviceToHost, m.stream));
        m.check_status();
    } catch (...) {
        cudaStreamSynchronize(m.stream);
        if (dx) cudaFree(dx);
        if (dy) cudaFree(dy);
        while (m.allocs.size() > first_alloc) {
            cudaFree(m.allocs.back());
            m.allocs.pop_back();
        }
        throw;
    }
    cudaFree(dx);
    cudaFree(dy);
    while (m.allocs.size() > first_alloc) {
        cudaFree(m.allocs.back());
        m.allocs.pop_back();
    }
}

// ------------------------------------------------------------------------------------------------
// Sampling without any allocation.  Some callers must not allocate device memory at the moment they
// sample: code running inside a memory-pool or arena discipline that forbids cudaMalloc on the hot
// path, latency-critical serving loops (cudaMalloc/cudaFree synchronise the device), and plugins that
// are handed device buffers by a host framework and may not own allocations of their own.  For them
// the sampler's work area lives in two file-scope device arrays that every GPU loading this library
// holds until the process exits: 2 x 4 MiB (kStaticSampleMaxElems floats + as many u32).
// ------------------------------------------------------------------------------------------------
constexpr size_t kStaticSampleMaxElems = size_t(1) << 20;  // rows * V <= 1,048,576 (e.g. 16 rows of a 65536 vocabulary)
static __device__ __align__(256) float g_static_sample_temp[kStaticSampleMaxElems];
static __device__ __align__(256) uint32_t g_static_sample_cnt[kStaticSampleMaxElems];

namespace {
struct StaticScratch {
    float* temp = nullptr;
    uint32_t* cnt = nullptr;
};
constexpr int kMaxDevices = 64;
StaticScratch g_static_scratch[kMaxDevices];
std::once_flag g_static_once[kMaxDevices];
}  // namespace

void set_last_error(const std::string& msg);  // defined with the C ABI

}  // namespace rsv

// The sampling kernel with its work area in static device memory; device pointers in, device pointer out.
// See include/rsv_b200.h for the contract.
extern "C" int rsv_op_sample_static(int device, void* stream, const float* logits_dev, int64_t rows, int64_t V, const float* sampler8_dev,
                                    const uint32_t* hist_dev, int64_t hist_stride, uint32_t* out_dev) {
    using namespace rsv;
    try {
        if (!logits_dev || !sampler8_dev || !out_dev) throw std::runtime_error("sample_static: null argument");
        if (rows < 1 || V < 1) throw std::runtime_error("sample_static: empty input");
        if (hist_stride < 0 || (hist_stride > 0 && !hist_dev)) throw std::runtime_error("sample_static: history is null but hist_stride > 0");
        if (hist_stride > 0x7fffffffLL || rows > 0x7fffffffLL || V > 0x7fffffffLL) throw std::runtime_error("sample_static: rows, V and hist_stride must fit in 31 bits");
        if ((uint64_t)rows * (uint64_t)V > kStaticSampleMaxElems)
            throw std::runtime_error("sample_static: rows * V = " + std::to_string((uint64_t)rows * (uint64_t)V) + " exceeds the static work area of " +
                                     std::to_string(kStaticSampleMaxElems) + " elements; use rsv_op_sample or fewer rows per call");
        if (device < 0 || device >= kMaxDevices) throw std::runtime_error("sample_static: device index out of range");
        RSV_CUDA(cudaSetDevice(device));
        StaticScratch& sc = g_static_scratch[device];
        // first call on this device: resolve the device addresses of the static arrays (in host code their names are only
        // handles, not device pointers).  Once per device, also when several host threads make their first call together.
        std::call_once(g_static_once[device], [&] {
            float* t = nullptr;
            uint32_t* c = nullptr;
            if (cudaGetSymbolAddress((void**)&t, g_static_sample_temp) == cudaSuccess && cudaGetSymbolAddress((void**)&c, g_static_sample_cnt) == cudaSuccess) {
                sc.cnt = c;
                sc.temp = t;
            }
        });
        if (!sc.temp || !sc.cnt) throw CudaError("sample_static: cudaGetSymbolAddress failed for the static work area");
        launch_sample((cudaStream_t)stream, logits_dev, (int)rows, (int)V, sampler8_dev, hist_stride ? hist_dev : nullptr, (int)hist_stride, nullptr, sc.temp, sc.cnt,
                      out_dev, nullptr, nullptr, 0, nullptr);
        return 0;
    } catch (const CudaError& e) {
        set_last_error(e.what());
        return 2;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return 1;
    }
}
