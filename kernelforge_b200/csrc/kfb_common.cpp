// Host-side helpers of libkfb: error reporting, scratch buffers, label
// bucketing and derivative offsets.
#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "kfb_internal.h"

namespace kfb {

static thread_local std::string g_last_error;

kfb_status set_error(kfb_status st, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return st;
}

const char *last_error() { return g_last_error.c_str(); }

// The device's default memory pool returns unused memory to the driver at every
// synchronisation unless told otherwise; the solves synchronise between
// iterations, so their scratch (hundreds of MB) would be unmapped and mapped
// again on every call, and the derivative kernels' chunk buffers (tens of GB on
// a 180 GB device) would be remapped per call.  Keep up to KFB_POOL_KEEP_GB
// (default 64) GB in the pool.
static void keep_pool_memory() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return;
    done[dev] = true;
    const char *v = std::getenv("KFB_POOL_KEEP_GB");
    const double gb = v ? std::atof(v) : 64.0;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return;
    }
    unsigned long long keep = (unsigned long long)((gb > 0 ? gb : 0.0) * (double)(1ull << 30));
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess)
        (void)cudaGetLastError();
}

kfb_status DevBuf::alloc(size_t nbytes, cudaStream_t s) {
    release();
    keep_pool_memory();
    stream = s;
    bytes = nbytes ? nbytes : 16;
    cudaError_t e = cudaMallocAsync(&ptr, bytes, s);
    if (e != cudaSuccess) {
        ptr = nullptr;
        (void)cudaGetLastError();
        return set_error(KFB_ERR_ALLOC, "cudaMallocAsync(%zu bytes) failed: %s", bytes,
                         cudaGetErrorString(e));
    }
    return KFB_OK;
}

void DevBuf::release() {
    if (ptr) cudaFreeAsync(ptr, stream);
    ptr = nullptr;
    bytes = 0;
}

kfb_status trim_pool(cudaStream_t s) {
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    int dev = 0;
    cudaMemPool_t pool;
    KFB_CUDA_TRY(cudaGetDevice(&dev));
    KFB_CUDA_TRY(cudaDeviceGetDefaultMemPool(&pool, dev));
    KFB_CUDA_TRY(cudaMemPoolTrimTo(pool, 0));
    return KFB_OK;
}

// Labels are nuclear charges or element indices: small non-negative integers
// take a direct table, anything else a map.  Labels are numbered in the order
// they are met and sorted at the end.
namespace {

class LabelIndex {
public:
    LabelIndex() { std::fill(table_, table_ + TABLE, -1); }
    // number of label q, given a new one when it has none
    int number(int q) {
        const int l = (unsigned)q < (unsigned)TABLE ? table_[q] : -1;
        return l >= 0 ? l : find(q);
    }
    const std::vector<int> &labels() const { return labels_; }

private:
    int find(int q) {
        if (q < 0 || q >= TABLE) {
            const auto it = other_.find(q);
            if (it != other_.end()) return it->second;
            other_[q] = (int)labels_.size();
        } else {
            table_[q] = (int)labels_.size();
        }
        labels_.push_back(q);
        return (int)labels_.size() - 1;
    }
    static constexpr int TABLE = 512;
    int table_[TABLE];
    std::map<int, int> other_;
    std::vector<int> labels_;
};

// Scratch of a plan, kept per thread while it is small: a fresh array of this
// size is mapped and faulted in page by page on every call (0.4 ms of the
// 1.2 ms that 150,000 atoms took).
constexpr size_t PLAN_KEEP = (size_t)1 << 22;   // bytes

// Label number of every active atom of a set, in order, and the label counts.
void number_atoms(const SetView &v, LabelIndex &ix, std::vector<int> &num,
                  std::vector<int> &count) {
    num.resize((size_t)v.nm * v.ma);
    int *out = num.data();
    count.assign(ix.labels().size() + 1, 0);
    int *cnt = count.data();
    for (int m = 0; m < v.nm; ++m) {
        const int32_t *q = v.q + (size_t)m * v.ma;
        const int na = v.natoms(m);
        for (int i = 0; i < na; ++i) {
            const int l = ix.number(q[i]);
            if (l + 1 >= (int)count.size()) {
                count.resize(2 * (l + 2), 0);
                cnt = count.data();
            }
            ++cnt[l];
            *out++ = l;
        }
    }
}

void fill_buckets(const SetView &v, const std::vector<int> &labels, const std::vector<int> &order,
                  const std::vector<int> &num, std::vector<int> &count, Buckets &bk) {
    const int L = (int)labels.size();
    count.resize(std::max<size_t>(count.size(), L), 0);
    bk.labels.resize(L);
    bk.lab_start.assign(L + 1, 0);
    std::vector<int> fill(L);
    for (int s = 0; s < L; ++s) {
        bk.labels[s] = labels[order[s]];
        fill[order[s]] = bk.lab_start[s];
        bk.lab_start[s + 1] = bk.lab_start[s] + count[order[s]];
    }
    bk.src.resize(bk.lab_start[L]);
    int *src = bk.src.data(), *f = fill.data();
    const int *l = num.data();
    for (int m = 0; m < v.nm; ++m) {
        const int na = v.natoms(m), base = m * v.ma;
        for (int i = 0; i < na; ++i) src[f[*l++]++] = base + i;
    }
}

}  // namespace

std::vector<int> collect_labels(const SetView &a, const SetView *b) {
    LabelIndex ix;
    for (const SetView *v : {&a, b})
        for (int m = 0; v && m < v->nm; ++m) {
            const int32_t *q = v->q + (size_t)m * v->ma;
            const int na = v->natoms(m);
            for (int i = 0; i < na; ++i) ix.number(q[i]);
        }
    std::vector<int> out = ix.labels();
    std::sort(out.begin(), out.end());
    return out;
}

void plan_buckets(const SetView &a, const SetView *b, Buckets &ba, Buckets *bb) {
    static thread_local std::vector<int> num_a, num_b;
    LabelIndex ix;
    std::vector<int> count_a, count_b;
    number_atoms(a, ix, num_a, count_a);
    if (b) number_atoms(*b, ix, num_b, count_b);
    const std::vector<int> &labels = ix.labels();
    std::vector<int> order(labels.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return labels[x] < labels[y]; });
    fill_buckets(a, labels, order, num_a, count_a, ba);
    if (b) fill_buckets(*b, labels, order, num_b, count_b, *bb);
    for (std::vector<int> *n : {&num_a, &num_b})
        if (n->capacity() * sizeof(int) > PLAN_KEEP) std::vector<int>().swap(*n);
}

long long deriv_offsets(const SetView &s, std::vector<int> &offs) {
    offs.resize(s.nm + 1);
    long long acc = 0;
    for (int m = 0; m < s.nm; ++m) {
        offs[m] = (int)acc;
        acc += 3LL * s.natoms(m);
    }
    offs[s.nm] = (int)acc;
    return acc;
}

kfb_status zero(void *ptr, size_t bytes, cudaStream_t s) {
    if (bytes) KFB_CUDA_TRY(cudaMemsetAsync(ptr, 0, bytes, s));
    return KFB_OK;
}

int device_sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

static bool g_timing = false;
static thread_local double g_last_ms = 0.0;

bool timing_enabled() { return g_timing; }

KernelTimer::KernelTimer(cudaStream_t s) : stream(s) {
    if (!g_timing) return;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
}
KernelTimer::~KernelTimer() {
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
}
void KernelTimer::start() {
    if (t0) cudaEventRecord(t0, stream);
}
void KernelTimer::stop() {
    if (!t1) return;
    cudaEventRecord(t1, stream);
    cudaEventSynchronize(t1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, t0, t1);
    g_last_ms = ms;
}

double last_kernel_ms() { return g_last_ms; }
void set_timing(bool on) { g_timing = on; }

bool device_is_sm100() {
    int dev = 0, major = 0, minor = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
    return major == 10 && minor == 0;
}

int trace_level() {
    static const int lvl = [] {
        const char *v = std::getenv("KFB_TRACE");
        return v ? std::atoi(v) : 0;
    }();
    return lvl;
}

static thread_local std::string g_path_log;

void note_path(const char *name) {
    if (g_path_log.size() > 4096) return;
    if (!g_path_log.empty()) g_path_log += ',';
    g_path_log += name;
}

void path_log_clear() { g_path_log.clear(); }
const std::string &path_log() { return g_path_log; }

static double now_ms() {
    using namespace std::chrono;
    return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

TraceScope::TraceScope(const char *n, cudaStream_t s) : name(n), stream(s), level(trace_level()) {
    if (level <= 0) return;
    if (level >= 2) cudaStreamSynchronize(stream);
    t0 = now_ms();
}

TraceScope::~TraceScope() {
    if (level <= 0) return;
    if (level >= 2) cudaStreamSynchronize(stream);
    std::fprintf(stderr, "[kfb-trace] %-28s %9.3f ms\n", name, now_ms() - t0);
}

}  // namespace kfb
