// librfk runtime: NVRTC flame kernels, render states, image steps, C ABI.
//
// Host-side counterpart of flame_compiler / flame_kernel / tonemapper
// (src/librefrakt/src/flame_compiler.cpp, src/librefrakt/src/image/tonemapper.cpp),
// using the CUDA runtime for memory and streams and the driver API for the
// NVRTC-built modules. Failures return a status with a thread-local message
// instead of logging and exiting.
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

#include "../../../include/rfk.h"
#include "../kernels/image_kernels.h"
#include "codegen.h"
#include "flamedb.h"
#include "genome.h"
#include "runtime_internal.h"

extern const char* const rfk_src_device;
extern const char* const rfk_src_iterate;

namespace {
thread_local std::string g_error;
}  // namespace

std::string& rfk::rt::error_message() { return g_error; }

using namespace rfk::rt;

namespace {

// Host mirror of rfk_chains / rfk_bin_args / rfk_counters in rfk_iterate.cuh.
struct dev_chains {
    float* x;
    float* y;
    float* c;
    unsigned char* last;
};
struct dev_bin_args {
    const float* samples;
    dev_chains st;
    float4* bins;
    unsigned w, h;
    unsigned seed, salt;
    unsigned call_id;
    unsigned check;
    unsigned long long quality_target;
    unsigned long long max_passes;
    unsigned long long time_ns;
    const volatile unsigned* stop;
    unsigned long long* counters;
    unsigned tmul;
    unsigned slice;
};
constexpr int kCounterWords = 6;
constexpr int kMaxTemporalMultiplier = 32;  // RFK_MAX_TMUL of rfk_iterate.cuh  // quality, passes, start, stop, draws, status|pad
constexpr uint32_t kMaxBinMillis = 60000;  // upper bound of one bin call

// Device buffers and events of one call, released on every exit path,
// including a failed check that throws.
struct call_scope {
    std::vector<void*> bufs;
    std::vector<cudaEvent_t> events;
    template <class T>
    T* alloc(size_t bytes, const char* what) {
        void* p = nullptr;
        cuda_check(cudaMalloc(&p, bytes), what);
        bufs.push_back(p);
        return static_cast<T*>(p);
    }
    cudaEvent_t event() {
        cudaEvent_t e = nullptr;
        cuda_check(cudaEventCreate(&e), "event");
        events.push_back(e);
        return e;
    }
    ~call_scope() {
        // on a failed check a launch of this call may still be reading them
        if (std::uncaught_exceptions() > 0) cudaDeviceSynchronize();
        for (void* p : bufs) cudaFree(p);
        for (cudaEvent_t e : events) cudaEventDestroy(e);
    }
};

// Stream-ordered temporaries of one call: allocated with cudaMallocAsync and
// released with cudaFreeAsync on the same stream on every exit path, so a
// check that throws between the allocations and the end of the call leaks
// nothing (the frees are ordered after whatever the call already queued).
struct stream_scope {
    cudaStream_t s;
    std::vector<void*> bufs;
    explicit stream_scope(cudaStream_t st) : s(st) {}
    template <class T>
    T* alloc(size_t bytes, const char* what) {
        void* p = nullptr;
        cuda_check(cudaMallocAsync(&p, bytes, s), what);
        bufs.push_back(p);
        return static_cast<T*>(p);
    }
    ~stream_scope() {
        for (void* p : bufs) cudaFreeAsync(p, s);
    }
};

// A state's way of its packed samples and temporal schedule to the device: pinned
// memory and device memory kept from one warm-up to the next, and one copy. With
// temporaries of each call (four stream-ordered allocations, three copies from
// pageable memory and a synchronisation for these) a state's re-warming for a 512 x 512
// preview takes 331 us, 105 of them in its kernels, and 125 this way; a new state
// is made in 0.08 ms less and destroyed in 0.09 ms more.
// The memory grows by half at least. What is outgrown goes back on the stream, pinned
// memory (cudaFreeHost waits for the whole device) with the state. The device part comes
// from the stream-ordered pool, as the temporaries did: taken from cudaMalloc it moved
// the histogram allocated after it to other physical pages, and where the hot pixels'
// lines fall in L2 changes a bin by up to a third (1080p bench flame: 95 G iterations/s
// here, 84 there).
struct sample_stage {
    char *host = nullptr, *dev = nullptr;
    size_t host_cap = 0, dev_cap = 0;
    std::vector<char*> outgrown;
    sample_stage() = default;
    sample_stage(const sample_stage&) = delete;
    ~sample_stage() {
        for (char* p : outgrown) cudaFreeHost(p);
        if (host) cudaFreeHost(host);
        if (dev) cudaFree(dev);
    }
    // Every copy and kernel that uses the memory has been waited for.
    void reserve(size_t host_bytes, size_t dev_bytes, cudaStream_t s) {
        if (host_bytes > host_cap) {
            outgrown.reserve(outgrown.size() + 1);
            char* p = nullptr;
            const size_t n = std::max(host_bytes, host_cap + host_cap / 2);
            cuda_check(cudaHostAlloc((void**)&p, n, cudaHostAllocDefault), "pinned samples");
            if (host) outgrown.push_back(host);
            host = p;
            host_cap = n;
        }
        if (dev_bytes > dev_cap) {
            char* p = nullptr;
            const size_t n = std::max(dev_bytes, dev_cap + dev_cap / 2);
            cuda_check(cudaMallocAsync((void**)&p, n, s), "alloc samples");
            if (dev) cudaFreeAsync(dev, s);
            dev = p;
            dev_cap = n;
        }
    }
};

// Waits for the stream when a check throws, so that nothing queued by the call
// still reads memory that the next one writes.
struct drain_on_throw {
    cudaStream_t s;
    ~drain_on_throw() {
        if (std::uncaught_exceptions() > 0) cudaStreamSynchronize(s);
    }
};

}  // namespace

struct rfk_state {
    sample_stage stage;
    std::shared_ptr<const kernel_impl> k;
    unsigned w = 0, h = 0, seed = 0;
    int grid = 0;
    int tmul = 1;  // temporal samples per persistent block
    size_t nchains = 0;
    float* d_samples = nullptr;
    float *d_x = nullptr, *d_y = nullptr, *d_c = nullptr;
    unsigned char* d_last = nullptr;
    float4* d_bins = nullptr;
    unsigned long long* d_counters = nullptr;  // kCounterWords + 98 (histogram + max density)
    unsigned long long* h_counters = nullptr;  // pinned mirror
    unsigned* h_stop = nullptr;                // mapped pinned
    unsigned* d_stop = nullptr;
    cudaEvent_t done = nullptr;
    bool own_bins = true;  // false: the caller's histogram (rfk_warmup_adopt)
    unsigned call_id = 0;
    double quality = 0.0;
    bool pending = false;

    ~rfk_state() {
        if (done) cudaEventSynchronize(done);
        for (void* p : {(void*)d_samples, (void*)d_x, (void*)d_y, (void*)d_c, (void*)d_last, (void*)d_counters})
            if (p) cudaFree(p);
        if (d_bins && own_bins) cudaFree(d_bins);
        if (h_counters) cudaFreeHost(h_counters);
        if (h_stop) cudaFreeHost(h_stop);
        if (done) cudaEventDestroy(done);
    }
};

namespace {

// Floats of a prepared parameter block: the reals (padded to even), the alias
// pick table (2 per xform, and 2 per xform pair with chaos), the palette
// (RFK_SAMPLE_FLOATS of rfk_iterate.cuh).
size_t sample_floats_for(const rfk::generated_flame& g) {
    size_t off = (g.size_reals + 1) / 2 * 2 + 2 * g.num_xforms;
    if (g.chaos) off += 2 * g.num_xforms * g.num_xforms;
    off = (off + 3) / 4 * 4;
    return off + 1024;
}

std::string full_source(const rfk::generated_flame& g) {
    std::ostringstream src;
    src << rfk_src_device << "\n" << g.source << "\n" << rfk_src_iterate << "\n";
    return src.str();
}

std::vector<char> nvrtc_build(const std::string& source, const std::string& arch_name, const rfk_compile_opts& o, int block,
                              int cpt, int flush, int sort, std::string& log, bool verbose = false) {
    const std::string arch = "--gpu-architecture=" + arch_name;
    const std::string d_block = "-DRFK_BLOCK=" + std::to_string(block);
    const std::string d_cpt = "-DRFK_CPT=" + std::to_string(cpt);
    const std::string d_flush = "-DRFK_FLUSH=" + std::to_string(flush);
    const std::string d_sort = "-DRFK_SORT=" + std::to_string(sort);
    // the compiler fits blocks_per_sm bin blocks per SM (registers capped
    // through the launch bounds); by default 40 resident warps: left alone,
    // it keeps kernel arguments and flame parameters in registers (about 80
    // per thread) and fewer blocks run
    const int minb = o.blocks_per_sm > 0 ? o.blocks_per_sm : std::max(1, 1280 / block);
    const std::string d_minb = "-DRFK_MINB=" + std::to_string(minb);
    std::vector<const char*> opts = {arch.c_str(), "-std=c++17", "-lineinfo", d_block.c_str(), d_cpt.c_str(),
                                     d_flush.c_str(), d_sort.c_str(), "-extra-device-vectorization"};
    opts.push_back(d_minb.c_str());
    if (verbose) opts.push_back("--ptxas-options=-v");  // per-kernel registers / spills / shared memory in the log
    if (!o.precise_math) {
        opts.push_back("--use_fast_math");
        opts.push_back("-DRFK_FAST_HYPOT=1");
    }
    nvrtcProgram prog;
    if (nvrtcCreateProgram(&prog, source.c_str(), "rfk_flame.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        fail(RFK_E_COMPILE, "nvrtcCreateProgram failed");
    nvrtcResult cr = nvrtcCompileProgram(prog, (int)opts.size(), opts.data());
    size_t log_size = 0;
    nvrtcGetProgramLogSize(prog, &log_size);
    std::string nlog(log_size, '\0');
    if (log_size) nvrtcGetProgramLog(prog, nlog.data());
    while (!nlog.empty() && nlog.back() == '\0') nlog.pop_back();
    log = nlog;
    if (cr != NVRTC_SUCCESS) {
        nvrtcDestroyProgram(&prog);
        fail(RFK_E_COMPILE, std::string("NVRTC: ") + nvrtcGetErrorString(cr) + "\n" + nlog);
    }
    size_t cubin_size = 0;
    nvrtcGetCUBINSize(prog, &cubin_size);
    std::vector<char> cubin(cubin_size);
    nvrtcGetCUBIN(prog, cubin.data());
    nvrtcDestroyProgram(&prog);
    return cubin;
}

// Sorting chains by xform pays off when there is more than one xform and the
// per-xform ballots stay few; sort = 0 in the options means the block sort.
int resolve_sort(const rfk_compile_opts& o, size_t nx) {
    const bool can = nx >= 2 && nx <= 32;
    if (o.sort < 0 || !can) return 0;
    return o.sort == 1 ? 1 : 2;
}

int resolve_cpt(const rfk_compile_opts& o, int sort) {
    if (o.chains_per_thread > 0) return o.chains_per_thread;
    return sort ? 4 : 1;
}

void check_options(const rfk_compile_opts& o) {
    const int block = o.block > 0 ? o.block : 256;
    if (block % 32 != 0 || block > 1024) fail(RFK_E_INVALID, "block must be a multiple of 32 up to 1024");
    if (o.chains_per_thread > 8 || o.chains_per_thread < 0) fail(RFK_E_INVALID, "chains_per_thread must be in [0, 8]");
    if (o.flush < 0 || o.flush > 4) fail(RFK_E_INVALID, "flush must be 0, 1, 2, 3 or 4");
    if (o.blocks_per_sm < 0 || o.blocks_per_sm > 32) fail(RFK_E_INVALID, "blocks_per_sm must be in [0, 32]");
    if (o.blocks_per_sm * block > 2048) fail(RFK_E_INVALID, "blocks_per_sm x block exceeds 2048 threads per SM");
}

// NVRTC module cache: (db hash, structure, options) -> kernel.
std::mutex g_cache_mu;
std::map<std::string, std::weak_ptr<kernel_impl>> g_cache;

std::shared_ptr<kernel_impl> compile(const rfk::flamedb& db, const rfk::flame& f, const rfk_compile_opts& o, std::string& log) {
    const auto t0 = std::chrono::steady_clock::now();
    auto k = std::make_shared<kernel_impl>();
    k->gen = rfk::generate_flame_code(db, f);
    check_options(o);
    k->block = o.block > 0 ? o.block : 256;
    k->sort = resolve_sort(o, k->gen.num_xforms);
    k->cpt = resolve_cpt(o, k->sort);
    k->flush = o.flush;
    check_options(o);
    k->sample_floats = sample_floats_for(k->gen);
    if (k->sample_floats * 4 > 44 * 1024) fail(RFK_E_INVALID, "flame too large for the shared-memory parameter block");
    k->salt = (uint32_t)(f.structure_hash() ^ (f.structure_hash() >> 32));

    k->source = full_source(k->gen);

    std::vector<char> cubin = nvrtc_build(k->source, device_arch(), o, k->block, k->cpt, k->flush, k->sort, log);
    cuda_check(cudaLibraryLoadData(&k->lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0), "cudaLibraryLoadData");
    cuda_check(cudaLibraryGetKernel(&k->f_prepare, k->lib, "rfk_prepare"), "rfk_prepare");
    cuda_check(cudaLibraryGetKernel(&k->f_warmup, k->lib, "rfk_warmup"), "rfk_warmup");
    cuda_check(cudaLibraryGetKernel(&k->f_bin, k->lib, "rfk_bin"), "rfk_bin");
    cuda_check(cudaLibraryGetKernel(&k->f_apply, k->lib, "rfk_apply"), "rfk_apply");
    cuda_check(cudaLibraryGetKernel(&k->f_bin_batch, k->lib, "rfk_bin_batch"), "rfk_bin_batch");
    cuda_check(cudaLibraryGetKernel(&k->f_bin_tm, k->lib, "rfk_bin_tm"), "rfk_bin_tm");
    cudaFuncAttributes fa{};
    cuda_check(cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(k->f_bin)), "attributes");
    k->regs = fa.numRegs;
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(k->f_bin), k->block, 0),
               "occupancy");
    if (per_sm < 1) fail(RFK_E_COMPILE, "bin kernel cannot be resident with block " + std::to_string(k->block));
    if (o.blocks_per_sm > 0) per_sm = std::min(per_sm, o.blocks_per_sm);
    k->grid = per_sm * device_sm_count();

    // weighted transcendental count per chain step
    double wsum = 0.0;
    for (auto& xf : f.xforms) wsum += xf.weight;
    double sfu = 0.0;
    for (size_t i = 0; i < f.xforms.size(); i++)
        sfu += (wsum > 0 ? f.xforms[i].weight / wsum : 0.0) * k->gen.xforms[i].sfu_ops;
    if (k->gen.has_final) sfu += k->gen.xforms.back().sfu_ops;
    k->sfu_per_iter = sfu;
    // affine FMAs per chain step: 4 per vlink affine (two per coordinate),
    // weighted like the transcendentals, plus the final xform's and the
    // screen projection's
    double fma = 4.0;
    for (size_t i = 0; i < f.xforms.size(); i++)
        fma += (wsum > 0 ? f.xforms[i].weight / wsum : 0.0) * 4.0 * k->gen.xforms[i].affines;
    if (k->gen.has_final) fma += 4.0 * k->gen.xforms.back().affines;
    k->fma_per_iter = fma;
    k->compile_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return k;
}

std::shared_ptr<kernel_impl> compile_cached(const rfk::flamedb& db, const rfk::flame& f, const rfk_compile_opts& o,
                                           std::string& log) {
    std::ostringstream key;
    key << db.hash() << "|" << f.structure_key() << "|" << o.precise_math << "," << o.block << "," << o.chains_per_thread
        << "," << o.flush << "," << o.blocks_per_sm << "," << o.sort;
    {
        std::lock_guard<std::mutex> lk(g_cache_mu);
        auto it = g_cache.find(key.str());
        if (it != g_cache.end())
            if (auto sp = it->second.lock()) return sp;
    }
    auto k = compile(db, f, o, log);
    std::lock_guard<std::mutex> lk(g_cache_mu);
    g_cache[key.str()] = k;
    return k;
}

// Temporal sample s of S: spline segment and t within it, as refactor.cu:266-270.
void temporal_schedule(unsigned S, unsigned nseg, std::vector<unsigned>& seg, std::vector<float>& t) {
    if (nseg == 0) fail(RFK_E_INVALID, "need at least 4 samples");
    if (S < nseg) fail(RFK_E_INVALID, "fewer temporal samples than spline segments");
    const unsigned seg_size = S / nseg;
    seg.resize(S);
    t.resize(S);
    for (unsigned s = 0; s < S; s++) {
        unsigned sg = s / seg_size;
        float tt = (float)(s % seg_size) / (float)(S / nseg);
        if (sg >= nseg) {
            sg = nseg - 1;
            tt = 1.0f;
        }
        seg[s] = sg;
        t[s] = tt;
    }
}

// Uploads samples (after fix_rotation) and the temporal schedule of nsmp samples
// through the state's memory, builds spline coefficients and runs the prepare kernel
// into d_out (nsmp x sample_floats), all on the stream: the caller waits for it
// before it returns, and on a throw (drain_on_throw).
void prepare_staged(sample_stage& st, const kernel_impl& k, const double* samples, size_t nsamples, unsigned nsmp,
                    unsigned seed, float* d_out, cudaStream_t s) {
    const size_t sample_size = k.gen.size_reals + rfk::palette_reals;
    if (nsamples < 4) fail(RFK_E_INVALID, "need at least 4 packed samples");
    const unsigned nseg = (unsigned)(nsamples - 3);
    std::vector<unsigned> seg;
    std::vector<float> t;
    temporal_schedule(nsmp, nseg, seg, t);
    std::vector<double> fixed(samples, samples + nsamples * sample_size);
    rfk::fix_rotation(fixed, sample_size, k.gen.size_reals, k.gen.affine_indices);
    const size_t b_samples = fixed.size() * sizeof(double), b_seg = nsmp * sizeof(unsigned);
    const size_t up = b_samples + 2 * b_seg, coeff_at = (up + 255) / 256 * 256;  // doubles, segments, t; then float4
    st.reserve(up, coeff_at + (size_t)nseg * sample_size * sizeof(float4), s);
    std::memcpy(st.host, fixed.data(), b_samples);
    std::memcpy(st.host + b_samples, seg.data(), b_seg);
    std::memcpy(st.host + b_samples + b_seg, t.data(), b_seg);
    const double* d_samples = reinterpret_cast<const double*>(st.dev);
    const unsigned* d_seg = reinterpret_cast<const unsigned*>(st.dev + b_samples);
    const float* d_t = reinterpret_cast<const float*>(st.dev + b_samples + b_seg);
    float4* d_coeff = reinterpret_cast<float4*>(st.dev + coeff_at);
    cuda_check(cudaMemcpyAsync(st.dev, st.host, up, cudaMemcpyHostToDevice, s), "H2D samples");
    cuda_check(rfk_launch_catmull(d_samples, (unsigned)sample_size, nseg, d_coeff, s), "catmull");
    unsigned ss = (unsigned)sample_size, salt = k.salt, jitter = 1;
    void* args[] = {&d_coeff, &ss, &d_seg, &d_t, &d_out, &seed, &salt, &jitter};
    launch(k.f_prepare, nsmp, 256, s, args, "rfk_prepare");
}

// Uploads samples (after fix_rotation), builds spline coefficients and runs
// the prepare kernel for the given schedule into d_out (count x sample_floats).
void prepare(const kernel_impl& k, const double* samples, size_t nsamples, const std::vector<unsigned>& seg,
             const std::vector<float>& t, unsigned seed, float* d_out, cudaStream_t s) {
    const size_t sample_size = k.gen.size_reals + rfk::palette_reals;
    if (nsamples < 4) fail(RFK_E_INVALID, "need at least 4 packed samples");
    std::vector<double> host(samples, samples + nsamples * sample_size);
    rfk::fix_rotation(host, sample_size, k.gen.size_reals, k.gen.affine_indices);
    const unsigned nseg = (unsigned)(nsamples - 3);
    for (unsigned sg : seg)
        if (sg >= nseg) fail(RFK_E_INVALID, "segment index out of range");
    stream_scope tmp(s);
    double* d_samples = tmp.alloc<double>(host.size() * sizeof(double), "alloc samples");
    float4* d_coeff = tmp.alloc<float4>((size_t)nseg * sample_size * sizeof(float4), "alloc coefficients");
    unsigned* d_seg = tmp.alloc<unsigned>(seg.size() * sizeof(unsigned), "alloc schedule");
    float* d_t = tmp.alloc<float>(t.size() * sizeof(float), "alloc schedule");
    cuda_check(cudaMemcpyAsync(d_samples, host.data(), host.size() * sizeof(double), cudaMemcpyHostToDevice, s), "H2D samples");
    cuda_check(cudaMemcpyAsync(d_seg, seg.data(), seg.size() * sizeof(unsigned), cudaMemcpyHostToDevice, s), "H2D schedule");
    cuda_check(cudaMemcpyAsync(d_t, t.data(), t.size() * sizeof(float), cudaMemcpyHostToDevice, s), "H2D schedule");
    cuda_check(rfk_launch_catmull(d_samples, (unsigned)sample_size, nseg, d_coeff, s), "catmull");
    unsigned ss = (unsigned)sample_size, salt = k.salt, jitter = 1;
    void* args[] = {&d_coeff, &ss, &d_seg, &d_t, &d_out, &seed, &salt, &jitter};
    launch(k.f_prepare, (unsigned)seg.size(), 256, s, args, "rfk_prepare");
    // the host vectors must outlive the copies
    cuda_check(cudaStreamSynchronize(s), "prepare");
}

void copy_out(char* buf, size_t cap, size_t* len, const std::string& s) {
    if (len) *len = s.size();
    if (buf && cap) {
        size_t n = std::min(cap - 1, s.size());
        std::memcpy(buf, s.data(), n);
        buf[n] = '\0';
    }
}

}  // namespace

// ====================================================================== C ABI
extern "C" {

const char* rfk_last_error(void) { return g_error.c_str(); }
int rfk_version(void) { return 100; }

rfk_status rfk_db_load(const char* dir, rfk_db** out) {
    return guard([&] {
        if (!dir || !out) fail(RFK_E_INVALID, "null argument");
        auto db = std::make_unique<rfk_db>();
        rfk::load_flamedb(db->db, dir);
        *out = db.release();
    });
}

void rfk_db_destroy(rfk_db* db) { delete db; }

int rfk_db_variation_count(const rfk_db* db) { return db ? (int)db->db.variations().size() : 0; }

rfk_status rfk_db_variation_name(const rfk_db* db, int index, char* buf, size_t cap) {
    return guard([&] {
        if (!db || index < 0 || index >= (int)db->db.variations().size()) fail(RFK_E_INVALID, "bad variation index");
        auto it = db->db.variations().begin();
        std::advance(it, index);
        copy_out(buf, cap, nullptr, it->first);
    });
}

uint64_t rfk_db_hash(const rfk_db* db) { return db ? db->db.hash() : 0; }

rfk_status rfk_db_add_variations(rfk_db* db, const char* yaml) {
    return guard([&] {
        if (!db || !yaml) fail(RFK_E_INVALID, "null argument");
        rfk::add_variations_yaml(db->db, yaml);
    });
}

rfk_status rfk_db_add_common(rfk_db* db, const char* name, const char* code) {
    return guard([&] {
        if (!db || !name || !code) fail(RFK_E_INVALID, "null argument");
        std::string err;
        if (!db->db.add_or_update_common(name, code, err)) fail(RFK_E_FORMAT, err);
    });
}

int rfk_db_remove_variation(rfk_db* db, const char* name) { return db && name && db->db.remove_variation(name) ? 1 : 0; }
int rfk_db_remove_common(rfk_db* db, const char* name) { return db && name && db->db.remove_common(name) ? 1 : 0; }
int rfk_db_is_variation(const rfk_db* db, const char* name) { return db && name && db->db.is_variation(name) ? 1 : 0; }
int rfk_db_is_parameter(const rfk_db* db, const char* v, const char* p) {
    return db && v && p && db->db.is_parameter(v, p) ? 1 : 0;
}
int rfk_db_is_common(const rfk_db* db, const char* name) { return db && name && db->db.is_common(name) ? 1 : 0; }

rfk_status rfk_db_variation_source(const rfk_db* db, const char* name, char* buf, size_t cap, size_t* len) {
    return guard([&] {
        if (!db || !name) fail(RFK_E_INVALID, "null argument");
        if (!db->db.is_variation(name)) fail(RFK_E_INVALID, std::string("unknown variation ") + name);
        const auto& def = db->db.get_variation(name);
        rfk::dsl::emit_env env;
        env.variation = name;
        for (auto& [pn, _] : def.params) env.param_expr[pn] = "P_" + pn;
        std::string s = rfk::dsl::emit_body(*def.apply_ast, env);
        if (def.precalc_ast) {
            rfk::dsl::emit_env penv = env;
            penv.precalc = true;
            s += "// precalc\n" + rfk::dsl::emit_body(*def.precalc_ast, penv);
        }
        copy_out(buf, cap, len, s);
    });
}

rfk_status rfk_flame_from_json(const rfk_db* db, const char* json, rfk_flame** out) {
    return guard([&] {
        if (!db || !json || !out) fail(RFK_E_INVALID, "null argument");
        auto f = std::make_unique<rfk_flame>();
        f->f = rfk::flame_from_json(db->db, rfk::parse_json(json));
        *out = f.release();
    });
}

rfk_status rfk_flame_from_flam3(const rfk_db* db, const char* xml, rfk_flame** out) {
    return guard([&] {
        if (!db || !xml || !out) fail(RFK_E_INVALID, "null argument");
        auto f = std::make_unique<rfk_flame>();
        f->f = rfk::flame_from_flam3(db->db, xml);
        *out = f.release();
    });
}

rfk_status rfk_flame_to_json(const rfk_flame* f, char* buf, size_t cap, size_t* len) {
    return guard([&] {
        if (!f) fail(RFK_E_INVALID, "null flame");
        copy_out(buf, cap, len, rfk::write_json(rfk::flame_to_json(f->f)));
    });
}

void rfk_flame_destroy(rfk_flame* f) { delete f; }

size_t rfk_flame_size_reals(const rfk_flame* f) { return f ? f->f.size_reals() : 0; }

rfk_status rfk_flame_pack_sample(const rfk_flame* f, int w, int h, double* out, size_t cap) {
    return guard([&] {
        if (!f || !out) fail(RFK_E_INVALID, "null argument");
        if (w <= 0 || h <= 0) fail(RFK_E_INVALID, "image size must be positive");
        std::vector<double> v;
        f->f.pack_sample(v, w, h);
        if (cap < v.size()) fail(RFK_E_INVALID, "output buffer too small: need " + std::to_string(v.size()));
        std::memcpy(out, v.data(), v.size() * sizeof(double));
    });
}

rfk_status rfk_flame_affine_indices(const rfk_flame* f, size_t* out, size_t cap, size_t* count) {
    return guard([&] {
        if (!f) fail(RFK_E_INVALID, "null flame");
        auto v = f->f.affine_indices();
        if (count) *count = v.size();
        if (out) {
            if (cap < v.size()) fail(RFK_E_INVALID, "output buffer too small");
            std::copy(v.begin(), v.end(), out);
        }
    });
}

rfk_status rfk_flame_tonemap_params(const rfk_flame* f, double out[4]) {
    return guard([&] {
        if (!f || !out) fail(RFK_E_INVALID, "null argument");
        out[0] = f->f.gamma;
        out[1] = f->f.brightness;
        out[2] = f->f.vibrancy;
        out[3] = f->f.highlight_power;
    });
}

uint64_t rfk_flame_structure_hash(const rfk_flame* f) { return f ? f->f.structure_hash() : 0; }

rfk_status rfk_compile(const rfk_db* db, const rfk_flame* f, const rfk_compile_opts* opts, rfk_kernel** out, char* log,
                       size_t log_cap) {
    std::string nlog;
    rfk_status st = guard([&] {
        if (!db || !f || !out) fail(RFK_E_INVALID, "null argument");
        rfk_compile_opts o{};
        if (opts) o = *opts;
        auto k = compile_cached(db->db, f->f, o, nlog);
        // handles share the cached module
        *out = new rfk_kernel{k};
    });
    if (log && log_cap) copy_out(log, log_cap, nullptr, st == RFK_OK ? nlog : g_error);
    return st;
}

}  // extern "C"

namespace {
const kernel_impl& K(const rfk_kernel* h) {
    if (!h || !h->impl) fail(RFK_E_INVALID, "null kernel");
    return *h->impl;
}
std::shared_ptr<kernel_impl> Kshared(const rfk_kernel* h) {
    if (!h || !h->impl) fail(RFK_E_INVALID, "null kernel");
    return h->impl;
}
}  // namespace

extern "C" {

void rfk_kernel_destroy(rfk_kernel* k) { delete k; }

rfk_status rfk_generate_source(const rfk_db* db, const rfk_flame* f, char* buf, size_t cap, size_t* len) {
    return guard([&] {
        if (!db || !f) fail(RFK_E_INVALID, "null argument");
        copy_out(buf, cap, len, full_source(rfk::generate_flame_code(db->db, f->f)));
    });
}

rfk_status rfk_compile_check(const rfk_db* db, const rfk_flame* f, const rfk_compile_opts* opts, const char* arch, char* log,
                             size_t log_cap) {
    std::string nlog;
    rfk_status st = guard([&] {
        if (!db || !f || !arch) fail(RFK_E_INVALID, "null argument");
        rfk_compile_opts o{};
        if (opts) o = *opts;
        check_options(o);
        auto g = rfk::generate_flame_code(db->db, f->f);
        const int sort = resolve_sort(o, g.num_xforms);
        nvrtc_build(full_source(g), arch, o, o.block > 0 ? o.block : 256, resolve_cpt(o, sort), o.flush, sort, nlog, true);
    });
    if (log && log_cap) copy_out(log, log_cap, nullptr, st == RFK_OK ? nlog : g_error);
    return st;
}

rfk_status rfk_kernel_get_info(const rfk_kernel* kh, rfk_kernel_info* out) {
    return guard([&] {
        const kernel_impl& k = K(kh);
        if (!out) fail(RFK_E_INVALID, "null output");
        out->grid = k.grid;
        out->block = k.block;
        out->chains_per_thread = k.cpt;
        out->flush = k.flush;
        out->sort = k.sort;
        out->registers = k.regs;
        out->num_xforms = (int)k.gen.num_xforms;
        out->has_final = k.gen.has_final;
        out->chaos = k.gen.chaos;
        out->size_reals = k.gen.size_reals;
        out->sample_floats = k.sample_floats;
        out->compile_ms = k.compile_ms;
        out->sfu_per_iter = k.sfu_per_iter;
        out->fma_per_iter = k.fma_per_iter;
    });
}

rfk_status rfk_kernel_source(const rfk_kernel* kh, char* buf, size_t cap, size_t* len) {
    return guard([&] { copy_out(buf, cap, len, K(kh).gen.source); });
}

namespace {
// Both warm-up entry points: a fresh cleared histogram (adopt == nullptr), or
// the caller's histogram taken as it is (flame_compiler.cpp:1037-1101 does
// not clear an adopted image; the dims overload at :1103-1108 clears its own).
rfk_status warmup_impl(const rfk_kernel* kh, const double* samples, size_t nsamples, float4* adopt, uint32_t w,
                       uint32_t h, uint32_t seed, uint32_t warmup_count, int temporal_multiplier, void* stream,
                       rfk_state** out) {
    return guard([&] {
        auto k = Kshared(kh);
        if (!samples || !out) fail(RFK_E_INVALID, "null argument");
        if (adopt && reinterpret_cast<uintptr_t>(adopt) % 16 != 0) fail(RFK_E_INVALID, "histogram must be 16-byte aligned");
        if (w == 0 || h == 0) fail(RFK_E_INVALID, "image size must be positive");
        if ((uint64_t)w * h > (1ull << 31)) fail(RFK_E_INVALID, "image too large");
        if (temporal_multiplier < 1 || temporal_multiplier > kMaxTemporalMultiplier)
            fail(RFK_E_INVALID, "temporal_multiplier must be in [1, 32]");
        cudaStream_t s = (cudaStream_t)stream;
        auto st = std::make_unique<rfk_state>();
        st->k = k;
        st->w = w;
        st->h = h;
        st->seed = seed;
        st->grid = k->grid;
        st->tmul = temporal_multiplier;
        // T x grid temporal samples, each with its own parameter block and chains
        const unsigned nsmp = (unsigned)st->grid * (unsigned)temporal_multiplier;
        st->nchains = (size_t)nsmp * k->block * k->cpt;
        cuda_check(cudaMalloc(&st->d_samples, (size_t)nsmp * k->sample_floats * sizeof(float)), "alloc samples");
        drain_on_throw drain{s};
        prepare_staged(st->stage, *k, samples, nsamples, nsmp, seed, st->d_samples, s);
        cuda_check(cudaMalloc(&st->d_x, st->nchains * sizeof(float)), "alloc chains");
        cuda_check(cudaMalloc(&st->d_y, st->nchains * sizeof(float)), "alloc chains");
        cuda_check(cudaMalloc(&st->d_c, st->nchains * sizeof(float)), "alloc chains");
        cuda_check(cudaMalloc(&st->d_last, st->nchains), "alloc chains");
        cuda_check(cudaMemsetAsync(st->d_last, 255, st->nchains, s), "init chains");
        if (adopt) {
            st->d_bins = adopt;
            st->own_bins = false;
        } else {
            cuda_check(cudaMalloc(&st->d_bins, (size_t)w * h * sizeof(float4)), "alloc histogram");
            cuda_check(cudaMemsetAsync(st->d_bins, 0, (size_t)w * h * sizeof(float4), s), "clear histogram");
        }
        cuda_check(cudaMalloc(&st->d_counters, (kCounterWords + 98) * sizeof(unsigned long long)), "alloc counters");
        cuda_check(cudaMemsetAsync(st->d_counters, 0, (kCounterWords + 98) * sizeof(unsigned long long), s), "clear counters");
        cuda_check(cudaHostAlloc(&st->h_counters, (kCounterWords + 98) * sizeof(unsigned long long), cudaHostAllocDefault), "pinned");
        cuda_check(cudaHostAlloc(&st->h_stop, sizeof(unsigned), cudaHostAllocMapped), "stop flag");
        *st->h_stop = 0;
        cuda_check(cudaHostGetDevicePointer((void**)&st->d_stop, st->h_stop, 0), "stop flag");
        cuda_check(cudaEventCreateWithFlags(&st->done, cudaEventDisableTiming), "event");
        dev_chains ch{st->d_x, st->d_y, st->d_c, st->d_last};
        unsigned ww = w, hh = h, sd = seed, salt = k->salt, wc = warmup_count;
        void* args[] = {&st->d_samples, &ch, &ww, &hh, &sd, &salt, &wc};
        launch(k->f_warmup, nsmp, (unsigned)k->block, s, args, "rfk_warmup");
        cuda_check(cudaStreamSynchronize(s), "warmup");
        *out = st.release();
    });
}
}  // namespace

rfk_status rfk_warmup(const rfk_kernel* kh, const double* samples, size_t nsamples, uint32_t w, uint32_t h, uint32_t seed,
                      uint32_t warmup_count, int temporal_multiplier, void* stream, rfk_state** out) {
    return warmup_impl(kh, samples, nsamples, nullptr, w, h, seed, warmup_count, temporal_multiplier, stream, out);
}

rfk_status rfk_warmup_adopt(const rfk_kernel* kh, const double* samples, size_t nsamples, void* bins, uint32_t w,
                            uint32_t h, uint32_t seed, uint32_t warmup_count, int temporal_multiplier, void* stream,
                            rfk_state** out) {
    if (!bins) return guard([] { fail(RFK_E_INVALID, "null histogram"); });
    return warmup_impl(kh, samples, nsamples, static_cast<float4*>(bins), w, h, seed, warmup_count,
                       temporal_multiplier, stream, out);
}

void rfk_state_destroy(rfk_state* s) { delete s; }

rfk_status rfk_state_rewarm(rfk_state* st, const double* samples, size_t nsamples, uint32_t seed, uint32_t warmup_count,
                            int clear, void* stream) {
    return guard([&] {
        if (!st || !samples) fail(RFK_E_INVALID, "null argument");
        if (st->pending) fail(RFK_E_INVALID, "a bin call is pending on this state: call rfk_bin_wait first");
        const kernel_impl& k = *st->k;
        cudaStream_t s = (cudaStream_t)stream;
        const unsigned nsmp = (unsigned)st->grid * (unsigned)st->tmul;
        drain_on_throw drain{s};
        prepare_staged(st->stage, k, samples, nsamples, nsmp, seed, st->d_samples, s);
        if (clear) cuda_check(cudaMemsetAsync(st->d_bins, 0, (size_t)st->w * st->h * sizeof(float4), s), "clear histogram");
        cuda_check(cudaMemsetAsync(st->d_counters, 0, (kCounterWords + 98) * sizeof(unsigned long long), s), "clear counters");
        st->seed = seed;
        st->quality = 0.0;
        st->call_id = 0;
        dev_chains ch{st->d_x, st->d_y, st->d_c, st->d_last};
        unsigned ww = st->w, hh = st->h, sd = seed, salt = k.salt, wc = warmup_count;
        void* args[] = {&st->d_samples, &ch, &ww, &hh, &sd, &salt, &wc};
        launch(k.f_warmup, nsmp, (unsigned)k.block, s, args, "rfk_warmup");
        cuda_check(cudaStreamSynchronize(s), "warmup");
    });
}

rfk_status rfk_bin_async(rfk_state* st, const rfk_bailout* bo, void* stream) {
    return guard([&] {
        if (!st || !bo) fail(RFK_E_INVALID, "null argument");
        if (!(bo->quality >= 0.0)) fail(RFK_E_INVALID, "quality must be >= 0");
        if (bo->quality == 0.0 && bo->iters == 0 && bo->millis == 0)
            fail(RFK_E_INVALID, "bailout needs a quality, pass or time limit");
        // one call at a time per state: a second call would re-record the
        // completion event and overwrite the pinned counters of the first
        if (st->pending) fail(RFK_E_INVALID, "a bin call is pending on this state: call rfk_bin_wait first");
        const kernel_impl& k = *st->k;
        cudaStream_t s = (cudaStream_t)stream;
        // The stop flag is cleared here, on the host, before anything is
        // queued: an rfk_state_abort issued at any time after this call
        // returns reaches the launch, even when earlier work keeps the
        // stream busy (a clear queued on the stream could run after the
        // abort and wipe it out). No launch of this state reads the flag now:
        // the previous call has been waited for.
        *reinterpret_cast<volatile unsigned*>(st->h_stop) = 0u;
        cuda_check(rfk_launch_clear_counters(st->d_counters, kCounterWords + 98, s), "clear counters");
        dev_bin_args a{};
        a.samples = st->d_samples;
        a.st = {st->d_x, st->d_y, st->d_c, st->d_last};
        a.bins = st->d_bins;
        a.w = st->w;
        a.h = st->h;
        a.seed = st->seed;
        a.salt = k.salt;
        a.call_id = st->call_id++ % 0xFFF0u;
        const double pixels = (double)st->w * st->h;
        a.quality_target = bo->quality > 0 ? (unsigned long long)(bo->quality * pixels * 255.0) : 0ull;
        a.max_passes = bo->iters;
        // Passes between bailout checks: about 1/8 of the target per round of
        // all chains, so the overshoot stays near one round when the target is
        // small next to the chain count.
        const double chains = (double)st->nchains;
        double chk = a.quality_target ? (double)a.quality_target / (chains * 255.0 * 8.0) : 32.0;
        chk = std::min(32.0, std::max(1.0, std::floor(chk)));
        a.check = (unsigned)chk;
        // Every call carries a time budget so that a target the flame can never
        // reach (all draws off-screen) still ends: min(millis, kMaxBinMillis).
        const uint32_t ms = (bo->millis == 0 || bo->millis > kMaxBinMillis) ? kMaxBinMillis : bo->millis;
        a.time_ns = (unsigned long long)ms * 1000000ull;
        a.stop = st->d_stop;
        a.counters = st->d_counters;
        a.tmul = (unsigned)st->tmul;
        a.slice = bo->temporal_slicing ? bo->temporal_slicing : 100u;
        void* args[] = {&a};
        if (st->tmul > 1)
            launch(k.f_bin_tm, (unsigned)st->grid, (unsigned)k.block, s, args, "rfk_bin_tm");
        else
            launch(k.f_bin, (unsigned)st->grid, (unsigned)k.block, s, args, "rfk_bin");
        cuda_check(rfk_launch_density_histogram(st->d_bins, st->w * st->h, st->d_counters + kCounterWords,
                                                st->d_counters + kCounterWords + 97, s),
                   "density histogram");
        cuda_check(cudaMemcpyAsync(st->h_counters, st->d_counters, (kCounterWords + 98) * sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost, s),
                   "D2H counters");
        cuda_check(cudaEventRecord(st->done, s), "event");
        st->pending = true;
    });
}

rfk_status rfk_bin_wait(rfk_state* st, rfk_bin_result* out) {
    return guard([&] {
        if (!st) fail(RFK_E_INVALID, "null state");
        if (!st->pending) fail(RFK_E_INVALID, "no bin call pending");
        cuda_check(cudaEventSynchronize(st->done), "bin");
        st->pending = false;
        const unsigned long long* c = st->h_counters;
        const double pixels = (double)st->w * st->h;
        rfk_bin_result r{};
        r.quality = (double)c[0] / (pixels * 255.0);
        r.elapsed_ms = c[3] > c[2] ? (double)(c[3] - c[2]) / 1e6 : 0.0;
        r.total_passes = c[1];
        r.total_draws = c[0] / 255;
        r.total_bins = (uint64_t)pixels;
        r.passes_per_thread = (double)c[1] / ((double)st->grid * st->k->block);
        r.max_density = (double)c[kCounterWords + 97];
        r.draw_count = c[4];
        r.status = (uint32_t)(c[5] & 0xFFFFFFFFu);
        st->quality += r.quality;
        if (out) *out = r;
    });
}

rfk_status rfk_bin(rfk_state* st, const rfk_bailout* bo, void* stream, rfk_bin_result* out) {
    rfk_status s = rfk_bin_async(st, bo, stream);
    if (s != RFK_OK) return s;
    return rfk_bin_wait(st, out);
}

rfk_status rfk_state_abort(rfk_state* st) {
    return guard([&] {
        if (!st || !st->h_stop) fail(RFK_E_INVALID, "null state");
        *reinterpret_cast<volatile unsigned*>(st->h_stop) = 1u;
    });
}

float* rfk_state_bins(rfk_state* st) { return st ? reinterpret_cast<float*>(st->d_bins) : nullptr; }

double rfk_state_quality(const rfk_state* st) { return st ? st->quality : 0.0; }

rfk_status rfk_state_chains(rfk_state* st, float* x, float* y, float* c, size_t cap, size_t* count) {
    return guard([&] {
        if (!st) fail(RFK_E_INVALID, "null state");
        if (count) *count = st->nchains;
        if (!x && !y && !c) return;
        if (cap < st->nchains) fail(RFK_E_INVALID, "output buffers too small");
        cuda_check(cudaDeviceSynchronize(), "sync");
        if (x) cuda_check(cudaMemcpy(x, st->d_x, st->nchains * 4, cudaMemcpyDeviceToHost), "D2H");
        if (y) cuda_check(cudaMemcpy(y, st->d_y, st->nchains * 4, cudaMemcpyDeviceToHost), "D2H");
        if (c) cuda_check(cudaMemcpy(c, st->d_c, st->nchains * 4, cudaMemcpyDeviceToHost), "D2H");
    });
}

rfk_status rfk_state_samples(rfk_state* st, float* out, size_t cap, size_t* count) {
    return guard([&] {
        if (!st) fail(RFK_E_INVALID, "null state");
        const size_t n = (size_t)st->grid * st->tmul * st->k->sample_floats;
        if (count) *count = n;
        if (!out) return;
        if (cap < n) fail(RFK_E_INVALID, "output buffer too small");
        cuda_check(cudaDeviceSynchronize(), "sync");
        cuda_check(cudaMemcpy(out, st->d_samples, n * 4, cudaMemcpyDeviceToHost), "D2H");
    });
}

rfk_status rfk_apply_xform(const rfk_kernel* kh, const float* params, int xform, const float* in_xyc, size_t n,
                           float* out_xyco, uint32_t seed) {
    return guard([&] {
        const kernel_impl& k = K(kh);
        if (!params || !in_xyc || !out_xyco) fail(RFK_E_INVALID, "null argument");
        if (xform >= (int)k.gen.num_xforms || xform < -1 || (xform == -1 && !k.gen.has_final))
            fail(RFK_E_INVALID, "bad xform index");
        if (n == 0) return;
        if (n > (1u << 30)) fail(RFK_E_INVALID, "too many points");
        call_scope cs;
        float* dp = cs.alloc<float>(k.sample_floats * 4, "alloc");
        float* di = cs.alloc<float>(n * 12, "alloc");
        float* dout = cs.alloc<float>(n * 16, "alloc");
        cuda_check(cudaMemcpy(dp, params, k.sample_floats * 4, cudaMemcpyHostToDevice), "H2D");
        cuda_check(cudaMemcpy(di, in_xyc, n * 12, cudaMemcpyHostToDevice), "H2D");
        unsigned nn = (unsigned)n, sd = seed;
        int xf = xform;
        void* args[] = {&dp, &xf, &di, &dout, &nn, &sd};
        launch(k.f_apply, (unsigned)((n + 255) / 256), 256, nullptr, args, "rfk_apply");
        cuda_check(cudaMemcpy(out_xyco, dout, n * 16, cudaMemcpyDeviceToHost), "D2H");
    });
}

rfk_status rfk_prepare_samples(const rfk_kernel* kh, const double* samples, size_t nsamples, const uint32_t* seg,
                               const float* t, size_t count, uint32_t seed, float* out) {
    return guard([&] {
        const kernel_impl& k = K(kh);
        if (!samples || !seg || !t || !out) fail(RFK_E_INVALID, "null argument");
        if (count == 0) return;
        std::vector<unsigned> sg(seg, seg + count);
        std::vector<float> tt(t, t + count);
        call_scope cs;
        float* d = cs.alloc<float>(count * k.sample_floats * 4, "alloc");
        prepare(k, samples, nsamples, sg, tt, seed, d, nullptr);
        cuda_check(cudaMemcpy(out, d, count * k.sample_floats * 4, cudaMemcpyDeviceToHost), "D2H");
    });
}

rfk_status rfk_prepare_samples_noalloc(const rfk_kernel* kh, const double* samples, size_t nsamples, const uint32_t* seg,
                                       const float* t, size_t count, uint32_t seed, float* out) {
    return guard([&] {
        const kernel_impl& k = K(kh);
        if (!samples || !seg || !t || !out) fail(RFK_E_INVALID, "null argument");
        if (count == 0) return;
        if (nsamples < 4) fail(RFK_E_INVALID, "need at least 4 packed samples");
        const size_t ss = k.gen.size_reals + rfk::palette_reals;
        const size_t nseg = nsamples - 3;
        for (size_t i = 0; i < count; i++)
            if (seg[i] >= nseg) fail(RFK_E_INVALID, "segment index out of range");
        const size_t naff = k.gen.affine_indices.size();
        unsigned aff[1024];
        if (naff > 1024) fail(RFK_E_INVALID, "more than 1024 affines");
        for (size_t i = 0; i < naff; i++) aff[i] = (unsigned)k.gen.affine_indices[i];
        // scratch layout, each region 256-byte aligned
        auto up = [](size_t b) { return (b + 255) / 256 * 256; };
        const size_t b_samples = up(nsamples * ss * sizeof(double));
        const size_t b_coeff = up(nseg * ss * sizeof(float4));
        const size_t b_aff = up(naff * sizeof(unsigned));
        const size_t b_seg = up(count * sizeof(uint32_t));
        const size_t b_t = up(count * sizeof(float));
        const size_t b_out = up(count * k.sample_floats * sizeof(float));
        const size_t need = b_samples + b_coeff + b_aff + b_seg + b_t + b_out;
        void* base = nullptr;
        size_t cap = 0;
        cuda_check(rfk_noalloc_scratch_address(&base, &cap), "no-alloc scratch address");
        if (need > cap)
            fail(RFK_E_INVALID, "request needs " + std::to_string(need) + " bytes of device scratch; the no-alloc scratch holds " +
                                    std::to_string(cap));
        char* p = static_cast<char*>(base);
        double* d_samples = reinterpret_cast<double*>(p);
        float4* d_coeff = reinterpret_cast<float4*>(p + b_samples);
        unsigned* d_aff = reinterpret_cast<unsigned*>(p + b_samples + b_coeff);
        unsigned* d_seg = reinterpret_cast<unsigned*>(p + b_samples + b_coeff + b_aff);
        float* d_t = reinterpret_cast<float*>(p + b_samples + b_coeff + b_aff + b_seg);
        float* d_out = reinterpret_cast<float*>(p + b_samples + b_coeff + b_aff + b_seg + b_t);
        cudaStream_t s = nullptr;
        cuda_check(cudaMemcpyAsync(d_samples, samples, nsamples * ss * sizeof(double), cudaMemcpyHostToDevice, s), "H2D samples");
        cuda_check(cudaMemcpyAsync(d_aff, aff, naff * sizeof(unsigned), cudaMemcpyHostToDevice, s), "H2D affines");
        cuda_check(cudaMemcpyAsync(d_seg, seg, count * sizeof(uint32_t), cudaMemcpyHostToDevice, s), "H2D schedule");
        cuda_check(cudaMemcpyAsync(d_t, t, count * sizeof(float), cudaMemcpyHostToDevice, s), "H2D schedule");
        cuda_check(rfk_launch_fix_rotation(d_samples, (unsigned)nsamples, (unsigned)ss, (unsigned)k.gen.size_reals, d_aff,
                                           (unsigned)naff, s),
                   "fix_rotation");
        cuda_check(rfk_launch_catmull(d_samples, (unsigned)ss, (unsigned)nseg, d_coeff, s), "catmull");
        unsigned sz = (unsigned)ss, salt = k.salt, sd = seed, jitter = 1;
        void* args[] = {&d_coeff, &sz, &d_seg, &d_t, &d_out, &sd, &salt, &jitter};
        launch(k.f_prepare, (unsigned)count, 256, s, args, "rfk_prepare");
        cuda_check(cudaMemcpyAsync(out, d_out, count * k.sample_floats * sizeof(float), cudaMemcpyDeviceToHost, s), "D2H");
        cuda_check(cudaStreamSynchronize(s), "prepare");
    });
}

rfk_status rfk_tonemap(const float* bins, uint32_t w, uint32_t h, void* out, int format, const rfk_tonemap_args* a,
                       uint64_t* histogram, uint64_t* max_density, void* stream) {
    return guard([&] {
        if (!bins || !out || !a) fail(RFK_E_INVALID, "null argument");
        if (format < RFK_HALF3 || format > RFK_FLOAT4) fail(RFK_E_INVALID, "bad output format");
        if ((histogram == nullptr) != (max_density == nullptr)) fail(RFK_E_INVALID, "histogram and max_density go together");
        if (!(a->quality > 0.0)) fail(RFK_E_INVALID, "quality must be positive");
        if ((uint64_t)w * h > 0xFFFFFFFFull) fail(RFK_E_INVALID, "image too large");
        // host constant as tonemapper.cpp:52, in single precision
        const float scale_constant = std::pow(10.0f, -std::log10((float)a->quality) - 0.5f);
        cuda_check(rfk_launch_tonemap(reinterpret_cast<const float4*>(bins), w * h, out, format, a->precise, (float)a->gamma,
                                      scale_constant, (float)a->brightness, (float)a->vibrancy, (float)a->highlight_power,
                                      (unsigned long long*)histogram, (unsigned long long*)max_density, nullptr, 0.0,
                                      (cudaStream_t)stream),
                   "tonemap");
    });
}

rfk_status rfk_convert(const void* in, int in_format, void* out, int out_format, uint32_t w, uint32_t h, int flip_y,
                       int swap_channels, void* stream) {
    return guard([&] {
        if (!in || !out) fail(RFK_E_INVALID, "null argument");
        if (in_format != RFK_HALF3 && in_format != RFK_HALF4) fail(RFK_E_INVALID, "input must be RFK_HALF3 or RFK_HALF4");
        if (out_format != RFK_FLOAT3 && out_format != RFK_FLOAT4 && out_format != RFK_UCHAR3 && out_format != RFK_UCHAR4)
            fail(RFK_E_INVALID, "output must be RFK_FLOAT3, RFK_FLOAT4, RFK_UCHAR3 or RFK_UCHAR4");
        if ((uint64_t)w * h > 0xFFFFFFFFull) fail(RFK_E_INVALID, "image too large");
        cuda_check(rfk_launch_convert(in, in_format == RFK_HALF3 ? 3 : 4, out, out_format, w, h, flip_y, swap_channels,
                                      (cudaStream_t)stream),
                   "convert");
    });
}

rfk_status rfk_density_histogram(const float* bins, uint32_t count, uint64_t* histogram, uint64_t* max_density,
                                 void* stream) {
    return guard([&] {
        if (!bins || !histogram || !max_density) fail(RFK_E_INVALID, "null argument");
        cuda_check(rfk_launch_density_histogram(reinterpret_cast<const float4*>(bins), count, (unsigned long long*)histogram,
                                                (unsigned long long*)max_density, (cudaStream_t)stream),
                   "density histogram");
    });
}

rfk_status rfk_density_blur(const float* in, float* out, uint32_t w, uint32_t h, const rfk_de_args* a, void* stream) {
    return guard([&] {
        if (!in || !out || !a) fail(RFK_E_INVALID, "null argument");
        if (in == out) fail(RFK_E_INVALID, "density blur needs distinct input and output");
        if (!(a->max_radius >= 0.0) || a->max_radius > RFK_DE_MAX_RADIUS_CAP) fail(RFK_E_INVALID, "max_radius must be in [0, 9]");
        if (!(a->min_radius >= 0.0) || a->min_radius > a->max_radius) fail(RFK_E_INVALID, "min_radius must be in [0, max_radius]");
        if (!(a->curve >= 0.0)) fail(RFK_E_INVALID, "curve must be >= 0");
        cuda_check(rfk_launch_de_blur(reinterpret_cast<const float4*>(in), reinterpret_cast<float4*>(out), w, h, (float)a->max_radius,
                                      (float)a->min_radius, (float)a->curve, (cudaStream_t)stream),
                   "density blur");
    });
}

rfk_status rfk_catmull_coefficients(const double* samples, uint32_t sample_size, uint32_t nseg, float* coeff, void* stream) {
    return guard([&] {
        if (!samples || !coeff) fail(RFK_E_INVALID, "null argument");
        cuda_check(rfk_launch_catmull(samples, sample_size, nseg, reinterpret_cast<float4*>(coeff), (cudaStream_t)stream), "catmull");
    });
}

rfk_status rfk_fix_rotation(double* samples, size_t nsamples, size_t sample_size, size_t flame_size,
                            const size_t* affine_indices, size_t n_affine) {
    return guard([&] {
        if (!samples || (!affine_indices && n_affine)) fail(RFK_E_INVALID, "null argument");
        if (flame_size > sample_size) fail(RFK_E_INVALID, "flame_size > sample_size");
        for (size_t i = 0; i < n_affine; i++)
            if (affine_indices[i] + 6 > flame_size) fail(RFK_E_INVALID, "affine index out of range");
        std::vector<double> v(samples, samples + nsamples * sample_size);
        rfk::fix_rotation(v, sample_size, flame_size, std::vector<size_t>(affine_indices, affine_indices + n_affine));
        std::copy(v.begin(), v.end(), samples);
    });
}

rfk_status rfk_probe_red_v4(size_t bytes, uint32_t iters, double* ops_per_s) {
    return guard([&] {
        if (!ops_per_s || bytes < 16) fail(RFK_E_INVALID, "bad argument");
        call_scope cs;
        float4* buf = cs.alloc<float4>(bytes, "alloc");
        cuda_check(cudaMemset(buf, 0, bytes), "clear");
        const unsigned blocks = (unsigned)device_sm_count() * 8, threads = 256;
        cudaEvent_t a = cs.event(), b = cs.event();
        cuda_check(rfk_launch_red_v4_probe(buf, bytes / 16, iters, blocks, threads, nullptr), "probe");
        // the median of 5 timed launches: one launch of this size takes under
        // a millisecond, and single timings scattered by about 2%
        std::vector<float> times;
        for (int rep = 0; rep < 5; rep++) {
            cudaEventRecord(a);
            cuda_check(rfk_launch_red_v4_probe(buf, bytes / 16, iters, blocks, threads, nullptr), "probe");
            cudaEventRecord(b);
            cuda_check(cudaEventSynchronize(b), "probe");
            float ms = 0;
            cuda_check(cudaEventElapsedTime(&ms, a, b), "probe timing");
            times.push_back(ms);
        }
        std::sort(times.begin(), times.end());
        *ops_per_s = (double)blocks * threads * iters / (times[times.size() / 2] * 1e-3);
    });
}

rfk_status rfk_probe_pipe(int pipe, uint32_t iters, double* ops_per_s) {
    return guard([&] {
        if (!ops_per_s || (pipe != 0 && pipe != 1) || iters == 0) fail(RFK_E_INVALID, "bad argument");
        const unsigned blocks = (unsigned)device_sm_count() * 8, threads = 256;
        call_scope cs;
        float* buf = cs.alloc<float>((size_t)blocks * threads * sizeof(float), "alloc");
        cudaEvent_t a = cs.event(), b = cs.event();
        cuda_check(rfk_launch_pipe_probe(buf, iters, pipe, blocks, threads, nullptr), "probe");
        cudaEventRecord(a);
        cuda_check(rfk_launch_pipe_probe(buf, iters, pipe, blocks, threads, nullptr), "probe");
        cudaEventRecord(b);
        cuda_check(cudaEventSynchronize(b), "probe");
        float ms = 0;
        cuda_check(cudaEventElapsedTime(&ms, a, b), "probe timing");
        *ops_per_s = (double)blocks * threads * iters * 8.0 / (ms * 1e-3);
    });
}

// ---------------------------------------------------------------- autotune --
// Times candidate launch shapes and histogram-flush strategies on the flame
// itself (the best choice depends on how concentrated its draws are), and
// keeps the fastest per (database, structure, genome values, image size).
namespace {
std::mutex g_tune_mu;
std::map<std::string, std::pair<rfk_compile_opts, double>> g_tune_cache;
}  // namespace

rfk_status rfk_autotune(const rfk_db* db, const rfk_flame* f, const double* samples, size_t nsamples, uint32_t w, uint32_t h,
                        uint32_t passes, rfk_compile_opts* best, rfk_tune_report* report) {
    return guard([&] {
        if (!db || !f || !samples || !best) fail(RFK_E_INVALID, "null argument");
        if (passes == 0) passes = 256;
        const size_t ss = f->f.size_reals() + rfk::palette_reals;
        std::ostringstream key;
        key << db->db.hash() << "|" << f->f.structure_key() << "|" << w << "x" << h << "|" << passes << "|";
        uint64_t vh = 1469598103934665603ull;
        const unsigned char* bytes = reinterpret_cast<const unsigned char*>(samples);
        for (size_t i = 0; i < nsamples * ss * sizeof(double); i++) vh = (vh ^ bytes[i]) * 1099511628211ull;
        key << vh;
        {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            auto it = g_tune_cache.find(key.str());
            if (it != g_tune_cache.end()) {
                *best = it->second.first;
                if (report) {
                    report->candidates = 0;
                    report->best_iters_per_s = it->second.second;
                    report->worst_iters_per_s = it->second.second;
                }
                return;
            }
        }
        // Only strategies that add aggregated sums (flush 1, 2, 4) are
        // candidates. With one red.v4 per draw (flush 0, 3) a pixel that
        // reaches 2^24 keeps that value: adding an opacity of 1 is a tie that
        // rounds back to the even 2^24, and smaller opacities round away
        // entirely, so a long render of a flame with a few hot pixels loses
        // most of their draws. The 256-pass timing launches cannot tell
        // whether the caller's render will get there; callers that know
        // their pixels stay below 2^24 draws may still compile flush 0.
        struct cand { int block, cpt, flush, sort, minb; };
        const cand cands[] = {{256, 8, 4, 2, 4}, {256, 4, 4, 2, 5}, {128, 8, 4, 2, 8}, {256, 4, 4, 1, 5},
                              {128, 8, 1, 2, 8}, {256, 8, 1, 2, 4}, {256, 4, 1, 2, 4}, {256, 2, 1, 2, 6},
                              {128, 4, 1, 2, 12}, {256, 4, 2, 2, 5}, {256, 4, 1, 1, 5}};
        double best_rate = -1.0, worst_rate = 1e300;
        int n = 0;
        for (const cand& c : cands) {
            rfk_compile_opts o{};
            o.block = c.block;
            o.chains_per_thread = c.cpt;
            o.flush = c.flush;
            o.sort = c.sort;
            o.blocks_per_sm = c.minb;
            rfk_kernel* kh = nullptr;
            if (rfk_compile(db, f, &o, &kh, nullptr, 0) != RFK_OK) continue;
            rfk_state* st = nullptr;
            rfk_status ws = rfk_warmup(kh, samples, nsamples, w, h, 1, 20, 1, nullptr, &st);
            if (ws != RFK_OK) {
                rfk_kernel_destroy(kh);
                continue;
            }
            rfk_bailout bo{passes, 0, 0.0};
            rfk_bin_result r{};
            double rate = 0.0;
            if (rfk_bin(st, &bo, nullptr, &r) == RFK_OK && rfk_bin(st, &bo, nullptr, &r) == RFK_OK && r.elapsed_ms > 0)
                rate = (double)r.total_passes / (r.elapsed_ms * 1e-3);
            rfk_state_destroy(st);
            rfk_kernel_destroy(kh);
            if (rate <= 0) continue;
            n++;
            worst_rate = std::min(worst_rate, rate);
            if (rate > best_rate) {
                best_rate = rate;
                *best = o;
            }
        }
        if (n == 0) fail(RFK_E_CUDA, "no autotune candidate ran");
        if (report) {
            report->candidates = n;
            report->best_iters_per_s = best_rate;
            report->worst_iters_per_s = worst_rate;
        }
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[key.str()] = {*best, best_rate};
    });
}

int rfk_device_sm_count(void) {
    int n = 0;
    rfk_status s = guard([&] { n = device_sm_count(); });
    return s == RFK_OK ? n : 0;
}

}  // extern "C"
