// engine.cpp -- host side of the device-resident GWR engine.
#include "engine.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <numeric>
#include <thread>

#include "gw_kernels.h"
#include "golden.h"

namespace gwgpu {

void check(cudaError_t e, const char* what)
{
    if (e != cudaSuccess) throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

namespace {

// Position of cell (x, y) along the Hilbert curve over a 2^31 x 2^31 grid
// (Hilbert's space-filling curve, by the usual quadrant rotate-and-reflect
// recursion from the top bit down).  Unlike the Z-order curve it never jumps:
// consecutive cells are neighbours, so any run of consecutive points is
// spatially compact.
uint64_t hilbert_index(uint32_t x, uint32_t y)
{
    const uint32_t n = 1u << 31;
    uint64_t d = 0;
    for (uint32_t s = n >> 1; s > 0; s >>= 1) {
        const uint32_t rx = (x & s) ? 1u : 0u;
        const uint32_t ry = (y & s) ? 1u : 0u;
        d += (uint64_t)s * s * ((3u * rx) ^ ry);
        if (ry == 0) {
            if (rx == 1) {
                x = n - 1 - x;
                y = n - 1 - y;
            }
            const uint32_t tmp = x;
            x = y;
            y = tmp;
        }
    }
    return d;
}

// fn(begin, end) over [0, n) in contiguous chunks on the host's threads (at
// least `grain` items per chunk); the calling thread takes the first chunk.
template <class F>
void parallel_for(size_t n, size_t grain, F&& fn)
{
    const size_t T = std::max<size_t>(1, std::min<size_t>(std::thread::hardware_concurrency(), 64));
    const size_t chunks = std::min(T, (n + grain - 1) / std::max<size_t>(grain, 1));
    if (chunks <= 1) {
        fn((size_t)0, n);
        return;
    }
    const size_t step = (n + chunks - 1) / chunks;
    std::vector<std::thread> pool;
    for (size_t c = 1; c < chunks; c++) {
        const size_t b = c * step, e = std::min(n, b + step);
        if (b < e) pool.emplace_back([&fn, b, e] { fn(b, e); });
    }
    fn((size_t)0, std::min(n, step));
    for (auto& t : pool) t.join();
}

// Stable LSD radix sort of (key, index) pairs by key, 8 bits a pass (passes
// whose byte is the same for every key are skipped): for input in index
// order, the same permutation std::sort gives the pairs.
void radix_sort(std::vector<std::pair<uint64_t, int>>& a)
{
    const size_t n = a.size();
    std::vector<std::pair<uint64_t, int>> b(n);
    uint64_t all_or = 0, all_and = ~0ull;
    for (const auto& x : a) {
        all_or |= x.first;
        all_and &= x.first;
    }
    for (int shift = 0; shift < 64; shift += 8) {
        if ((((all_or ^ all_and) >> shift) & 0xff) == 0) continue;
        size_t cnt[257] = {};
        for (const auto& x : a) cnt[((x.first >> shift) & 0xff) + 1]++;
        for (int q = 0; q < 256; q++) cnt[q + 1] += cnt[q];
        for (const auto& x : a) b[cnt[(x.first >> shift) & 0xff]++] = x;
        a.swap(b);
    }
}

// FP64 unit vectors (cos lat cos lon, cos lat sin lon, sin lat) of points given
// in radians, as three arrays of n: the chord form of the great-circle
// distance, and the source of every geographic record and bound below.
std::vector<double> unit_vectors(const std::vector<double>& lonR, const std::vector<double>& latR)
{
    const size_t n = lonR.size();
    std::vector<double> e(3 * n);
    parallel_for(n, 4096, [&](size_t b, size_t en) {
        for (size_t s = b; s < en; s++) {
            const double cl = std::cos(latR[s]);
            e[s] = cl * std::cos(lonR[s]);
            e[n + s] = cl * std::sin(lonR[s]);
            e[2 * n + s] = std::sin(latR[s]);
        }
    });
    return e;
}

// Geographic bounds of consecutive tiles of `size` points (sorted order), from
// the points' unit vectors (3 x n).
std::vector<TileCap> make_caps(const std::vector<double>& e, int size)
{
    const int n = (int)(e.size() / 3), nt = (n + size - 1) / size;
    std::vector<TileCap> caps(nt);
    parallel_for((size_t)nt, 256, [&](size_t tb, size_t te) {
        for (int t = (int)tb; t < (int)te; t++) {
            const int s0 = t * size, s1 = std::min(n, s0 + size);
            double sx = 0, sy = 0, sz = 0;
            for (int s = s0; s < s1; s++) {
                sx += e[s];
                sy += e[(size_t)n + s];
                sz += e[2 * (size_t)n + s];
            }
            double nrm = std::sqrt(sx * sx + sy * sy + sz * sz);
            TileCap c{1.0, 0.0, 0.0, 2.0};  // degenerate tile: no bound
            if (nrm > 1e-12) {
                c = TileCap{sx / nrm, sy / nrm, sz / nrm, 0.0};
                for (int s = s0; s < s1; s++) {
                    const double dx = e[s] - c.cx, dy = e[(size_t)n + s] - c.cy, dz = e[2 * (size_t)n + s] - c.cz;
                    c.rho = std::max(c.rho, std::sqrt(dx * dx + dy * dy + dz * dz));
                }
                c.rho = c.rho * (1.0 + 1e-12) + 1e-15;
            }
            caps[t] = c;
        }
    });
    return caps;
}

// FP64 boxes of consecutive tiles of `size` points.
std::vector<TileBox> make_boxes(const std::vector<double>& hu, const std::vector<double>& hv, int size)
{
    const int n = (int)hu.size(), nt = (n + size - 1) / size;
    std::vector<TileBox> out(nt);
    for (int t = 0; t < nt; t++) {
        TileBox b{hu[t * size], hu[t * size], hv[t * size], hv[t * size]};
        for (int s = t * size; s < std::min(n, (t + 1) * size); s++) {
            b.ulo = std::min(b.ulo, hu[s]);
            b.uhi = std::max(b.uhi, hu[s]);
            b.vlo = std::min(b.vlo, hv[s]);
            b.vhi = std::max(b.vhi, hv[s]);
        }
        out[t] = b;
    }
    return out;
}

void split_fp32(double v, float& hi, float& lo)
{
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

// FP32 records of geographic points, padded to whole 32-point tiles: the unit vector (e:
// 3 x n) split hi/lo in two float4 (its z is sin(lat)).  Planar ones: k_planar_proxy.
std::vector<float4> point_records(const std::vector<double>& e)
{
    const size_t n = e.size() / 3, nt32 = (n + 31) / 32;
    std::vector<float4> pts(2 * nt32 * 32, make_float4(0.f, 0.f, 0.f, 0.f));
    parallel_for(n, 8192, [&](size_t b, size_t en) {
        for (size_t s = b; s < en; s++) {
            float xh, xl, yh, yl, zh, zl;
            split_fp32(e[s], xh, xl);
            split_fp32(e[n + s], yh, yl);
            split_fp32(e[2 * n + s], zh, zl);
            pts[2 * s] = make_float4(xh, yh, zh, 0.f);
            pts[2 * s + 1] = make_float4(xl, yl, zl, 0.f);
        }
    });
    return pts;
}

// FP32 caps of consecutive tiles of `size` geographic points, rounded outward.
std::vector<float4> tile_bounds(const std::vector<double>& e, int size)
{
    const std::vector<TileCap> cp = make_caps(e, size);
    std::vector<float4> tb(cp.size());
    for (size_t t = 0; t < cp.size(); t++)
        tb[t] = make_float4((float)cp[t].cx, (float)cp[t].cy, (float)cp[t].cz,
                            nextafterf((float)cp[t].rho, INFINITY) * (1.0f + 1e-6f) + 1e-7f);
    return tb;
}

// GWRBase::AICc (GWRBase.h:90-94) from RSS and tr(S).
double aicc(double n, double rss, double trS)
{
    return n * std::log(rss / n) + n * std::log(2 * M_PI) + n * ((n + trS) / (n - 2 - trS));
}

// The distance cache of each device, shared by the engines on it (see
// Engine::setDistanceCacheLimit).  Every launch that fills or reads it runs
// under `mu` and records `used` on its engine's stream; a new owner's stream
// waits for that event before it overwrites the buffer.
struct DeviceD2Cache {
    std::mutex mu;
    float* ptr = nullptr;
    size_t bytes = 0;
    const Engine* owner = nullptr;
    cudaEvent_t used = nullptr;
};
constexpr int kMaxDevices = 64;
// Allocated once and never destroyed, so engines that outlive static
// destruction at process exit still find their device's entry and mutex.
DeviceD2Cache* const g_d2c = new DeviceD2Cache[kMaxDevices];

DeviceD2Cache& device_d2c(int device)
{
    if (device < 0 || device >= kMaxDevices) throw std::invalid_argument("device ordinal out of range");
    return g_d2c[device];
}

// Frees the device's cache (the caller holds its lock); waits for its last use.
void free_d2c(DeviceD2Cache& c)
{
    if (c.used) cudaEventSynchronize(c.used);
    if (c.ptr) cudaFree(c.ptr);
    c.ptr = nullptr;
    c.bytes = 0;
    c.owner = nullptr;
}

// The kept weights of each device (Engine::takeWeights), with the engines alive on it.
struct DeviceWeights {
    std::mutex mu;
    std::condition_variable idle;
    unsigned long long* ptr = nullptr;
    size_t bytes = 0;
    const Engine* user = nullptr;  // between the passes of a call
    cudaEvent_t used = nullptr;    // the last user's last launch
    int engines = 0;
};
DeviceWeights* const g_weights = new DeviceWeights[kMaxDevices];

// (the caller holds the lock, and nobody uses the buffer)
void free_weights(DeviceWeights& w)
{
    if (w.ptr) {
        cudaEventSynchronize(w.used);
        cudaFree(w.ptr);
    }
    w.ptr = nullptr;
    w.bytes = 0;
}

}  // namespace

bool release_idle_scratch()
{
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return false;
    DeviceWeights& w = g_weights[device];
    std::lock_guard<std::mutex> lk(w.mu);
    if (w.user || !w.ptr) return false;
    free_weights(w);
    return true;
}

Engine::Engine(int device) : device_(device)
{
    check(cudaSetDevice(device), "cudaSetDevice");
    if (device >= kMaxDevices) throw std::invalid_argument("device ordinal out of range");
    cudaDeviceProp prop;
    check(cudaGetDeviceProperties(&prop, device), "cudaGetDeviceProperties");
    num_sms_ = prop.multiProcessorCount;
    check(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
    check(cudaMallocHost(&host_sums_, 8 * sizeof(double)), "cudaMallocHost");
    DeviceWeights& w = g_weights[device_];
    std::lock_guard<std::mutex> lk(w.mu);
    w.engines++;
}

Engine::~Engine()
{
    if (stream_) cudaStreamSynchronize(stream_);
    if (device_ >= 0 && device_ < kMaxDevices) {
        DeviceD2Cache& c = g_d2c[device_];
        std::lock_guard<std::mutex> lk(c.mu);
        if (c.owner == this) {
            cudaSetDevice(device_);
            free_d2c(c);
        }
    }
    {
        leaveWeights();
        DeviceWeights& w = g_weights[device_];
        std::lock_guard<std::mutex> lk(w.mu);
        if (--w.engines == 0) {
            cudaSetDevice(device_);
            free_weights(w);
        }
    }
    for (auto& e : events_)
        if (e) cudaEventDestroy(e);
    for (auto& pt : pending_) {
        cudaEventDestroy(pt.e0);
        cudaEventDestroy(pt.e1);
    }
    if (host_sums_) cudaFreeHost(host_sums_);
    if (stream_) cudaStreamDestroy(stream_);
}

void Engine::synchronize() { check(cudaStreamSynchronize(stream_), "cudaStreamSynchronize"); }

DevPoints Engine::points() const
{
    DevPoints P;
    P.n = n_;
    P.u = u_.get();
    P.v = v_.get();
    P.uR = uR_.get();
    P.vR = vR_.get();
    P.e = e_.get();
    return P;
}


void Engine::setData(int n, int p, const double* x, const double* y, const double* coords, bool geographic)
{
    if (n < 2) throw std::invalid_argument("GWRBasic needs at least two data points");
    if (p < 1 || p > kMaxP) throw std::invalid_argument("number of independent variables must be in [1, 32]");
    check(cudaSetDevice(device_), "cudaSetDevice");
    n_ = n;
    p_ = p;
    mm_ = p * (p + 1) / 2;
    m_ = mm_ + p;
    geographic_ = geographic;
    thr_valid_ = false;
    gall_valid_ = false;
    mixed_ready_ = false;
    ixy_tried_ = ixy_ok_ = zfx_ready_ = false;

    // Hilbert order of the coordinates
    double umin = coords[0], umax = coords[0], vmin = coords[n], vmax = coords[n];
    for (int i = 0; i < n; i++) {
        umin = std::min(umin, coords[i]);
        umax = std::max(umax, coords[i]);
        vmin = std::min(vmin, coords[n + i]);
        vmax = std::max(vmax, coords[n + i]);
    }
    const double su = umax > umin ? 2147483647.0 / (umax - umin) : 0.0;
    const double sv = vmax > vmin ? 2147483647.0 / (vmax - vmin) : 0.0;
    // the raw data go up as they are; order and gather happen on the device
    const int ntiles = (n + kTile - 1) / kTile;
    raw_.alloc((size_t)n * (p + 3));
    double* rx = raw_.get() + 2 * (size_t)n;
    double* ry = rx + (size_t)n * p;
    check(cudaMemcpyAsync(raw_.get(), coords, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, stream_), "H2D coords");
    d_perm_.alloc(n);
    orderPoints(n, coords, raw_.get(), umin, su, vmin, sv, d_perm_.get(), perm_);
    check(cudaMemcpyAsync(rx, x, sizeof(double) * (size_t)n * p, cudaMemcpyHostToDevice, stream_), "H2D x");
    check(cudaMemcpyAsync(ry, y, sizeof(double) * n, cudaMemcpyHostToDevice, stream_), "H2D y");
    if (geographic) {
        dhi_ = 20300.0;  // above half the WGS-84 meridian circumference with the flattening term
    } else {
        double du = umax - umin, dv = vmax - vmin;
        dhi_ = std::sqrt(du * du + dv * dv) * (1.0 + 1e-9);
        if (!(dhi_ > 0.0) || !std::isfinite(dhi_)) dhi_ = 1.0;
    }
    dlo_ = std::ldexp(dhi_, -24);

    u_.alloc(n);
    v_.alloc(n);
    if (geographic) {
        uR_.alloc(n);
        vR_.alloc(n);
    } else {
        uR_.clear();
        vR_.clear();
    }
    x_.alloc((size_t)n * p);
    y_.alloc(n);
    z_.alloc((size_t)n * m_);
    g_.alloc((size_t)n * m_);
    thr_.alloc(n);
    sel0_.alloc(n);
    sel1_.alloc(n);
    beta_.alloc((size_t)n * p);
    sii_.alloc(n);
    resid_.alloc(n);
    partials_.alloc(4096 * 4);
    tiles_.alloc(ntiles);
    key_.alloc(2);
    check(launch_gather_points(n, raw_.get(), d_perm_.get(), geographic, u_.get(), v_.get(), uR_.get(), vR_.get(), stream_),
          "gather points");
    check(launch_gather_xy(n, p, rx, ry, d_perm_.get(), x_.get(), y_.get(), stream_), "gather x, y");
    check(launch_build_z(n, p, x_.get(), y_.get(), z_.get(), stream_), "build_z");
    stats_.kernel_launches += 3;
    synchronize();  // perm_ is there
    hu_.resize(n);
    hv_.resize(n);
    std::vector<double> huR(geographic ? n : 0), hvR(geographic ? n : 0);
    const double DE2RA = M_PI / 180;
    parallel_for((size_t)n, 65536, [&](size_t b, size_t e) {
        for (size_t s = b; s < e; s++) {
            hu_[s] = coords[perm_[s]];
            hv_[s] = coords[(size_t)n + perm_[s]];
            if (geographic) {
                huR[s] = hu_[s] * DE2RA;
                hvR[s] = hv_[s] * DE2RA;
            }
        }
    });
    if (geographic) {
        he_ = unit_vectors(huR, hvR);
        e_.alloc(he_.size());
        check(cudaMemcpyAsync(e_.get(), he_.data(), sizeof(double) * he_.size(), cudaMemcpyHostToDevice, stream_),
              "H2D unit vectors");
        std::vector<TileBox> ht = make_boxes(hu_, hv_, kTile);
        check(cudaMemcpyAsync(tiles_.get(), ht.data(), sizeof(TileBox) * ntiles, cudaMemcpyHostToDevice, stream_),
              "H2D tiles");
        std::vector<TileCap> hc = make_caps(he_, kTile);
        caps_.alloc(hc.size());
        check(cudaMemcpyAsync(caps_.get(), hc.data(), sizeof(TileCap) * hc.size(), cudaMemcpyHostToDevice, stream_),
              "H2D caps");
        synchronize();
    } else {
        he_.clear();
        e_.clear();
        caps_.clear();
    }
    recycleRanks();
    hist_.clear();
    hist_tried_ = false;
    hist_valid_ = false;
    d2c_valid_ = false;
    buildProxy();
}


// perm (device and host): n points in Hilbert order, from `coords` on the device
// (`host`: the same on the host, for sizes below kPrepMin).
void Engine::orderPoints(int n, const double* host, const double* coords, double umin, double su, double vmin, double sv,
                         int* d_perm, std::vector<int>& perm)
{
    perm.resize(n);
    if (n >= kPrepMin) {
        prep_.alloc(hilbert_scratch_bytes(n));
        check(launch_hilbert_order(n, coords, umin, su, vmin, sv, prep_.get(), d_perm, stream_), "Hilbert order");
        stats_.kernel_launches += 25;
        check(cudaMemcpyAsync(perm.data(), d_perm, sizeof(int) * n, cudaMemcpyDeviceToHost, stream_), "D2H order");
        return;  // the caller synchronises before it reads perm
    }
    std::vector<std::pair<uint64_t, int>> keyed(n);
    for (int i = 0; i < n; i++) {
        const double fu = (host[i] - umin) * su, fv = (host[(size_t)n + i] - vmin) * sv;
        const uint32_t qu = std::isfinite(fu) ? (uint32_t)std::min(std::max(fu, 0.0), 2147483647.0) : 0u;
        const uint32_t qv = std::isfinite(fv) ? (uint32_t)std::min(std::max(fv, 0.0), 2147483647.0) : 0u;
        keyed[i] = {hilbert_index(qu, qv), i};
    }
    radix_sort(keyed);
    for (int s = 0; s < n; s++) perm[s] = keyed[s].second;
    check(cudaMemcpyAsync(d_perm, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, stream_), "H2D order");
}

void Engine::setVariables(int p, const double* x, const double* y)
{
    if (n_ == 0) throw std::logic_error("no data");
    if (p < 1 || p > kMaxP) throw std::invalid_argument("number of independent variables must be in [1, 32]");
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int n = n_;
    p_ = p;
    mm_ = p * (p + 1) / 2;
    m_ = mm_ + p;
    gall_valid_ = false;
    mixed_ready_ = false;
    zfx_ready_ = false;
    raw_.alloc((size_t)n * (p + 3));
    double* rx = raw_.get();
    double* ry = rx + (size_t)n * p;
    x_.alloc((size_t)n * p);
    z_.alloc((size_t)n * m_);
    g_.alloc((size_t)n * m_);
    beta_.alloc((size_t)n * p);
    rvec_.alloc((size_t)n * p);
    check(cudaMemcpyAsync(rx, x, sizeof(double) * (size_t)n * p, cudaMemcpyHostToDevice, stream_), "H2D x");
    check(cudaMemcpyAsync(ry, y, sizeof(double) * n, cudaMemcpyHostToDevice, stream_), "H2D y");
    check(launch_gather_xy(n, p, rx, ry, d_perm_.get(), x_.get(), y_.get(), stream_), "gather x, y");
    stats_.kernel_launches += 1;
    check(launch_build_z(n, p, x_.get(), y_.get(), z_.get(), stream_), "build_z");
    stats_.kernel_launches += 1;
    synchronize();
}

void Engine::fitDevice(double bw, bool adaptive, int kernel, bool se, double* ainv)
{
    if (n_ == 0) throw std::logic_error("no data");
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int n = n_, p = p_;
    const int saved = precision_;
    precision_ = kFP64;
    struct Restore {
        int& slot;
        int value;
        double*& out;
        ~Restore()
        {
            slot = value;
            out = nullptr;
        }
    } restore{precision_, saved, ainv_out_};
    g2_.alloc((size_t)n * mm_);
    vvec_.alloc((size_t)n * p);
    bse_.alloc((size_t)n * p);
    qdiag_.alloc(n);
    computeThresholds(bw, adaptive);
    {
        WeightScope scope{*this};
        contract(z_.get(), m_, g_.get(), m_, bw, adaptive, kernel, false, 1, se ? WeightUse::kKept : WeightUse::kOnce);
        if (se) contract(z_.get(), mm_, g2_.get(), mm_, bw, adaptive, kernel, false, 2, WeightUse::kAgain);
    }
    if (!se)  // the solve still forms the (unused) SE terms from G2
        check(cudaMemsetAsync(g2_.get(), 0, sizeof(double) * g2_.size(), stream_), "memset G2");
    ainv_out_ = ainv;
    double s[4];
    solve(kSolveFit, bw, adaptive, kernel, s);
    if (s[3] > 0.0) throw NotSPDError("inv_sympd(): matrix is singular or not positive definite");
}

// qdiag_ (and S) of the last FP64 fit-mode solve.
void Engine::hatPass(double bw, bool adaptive, int kernel, double* S, int row_target, double* s_row)
{
    HatArgs a{};
    a.P = points();
    a.tb16 = tb16_.get();
    a.tile_thr = tile_thr16_.get();
    a.X = x_.get();
    a.p = p_;
    a.v = vvec_.get();
    a.thr = thrPtr(adaptive);
    a.bw = bw;
    a.kernel = kernel;
    // v_i = A_i^-1 x_i is large where a column rests on small weights: FP64 ones there too
    if (fxReady(bw, adaptive, kernel) && ixy_exact_ && !guard_hit_) {
        hat_rows_.alloc(n_);
        a.xy = geographic_ ? nullptr : ixy_.get();
        a.e3 = geographic_ ? ie3_.get() : nullptr;
        a.geo = geo_.get();
        a.rows = hat_rows_.get();
        stats_.kernel_launches += 1;
    }
    a.S = S;
    a.perm = d_perm_.get();
    a.row_target = row_target;
    a.s_row = s_row;
    const int nsplit = hat_splits(n_, num_sms_);
    hat_sum_.alloc((size_t)n_ * nsplit);
    a.qsum = hat_sum_.get();
    check(launch_hat_pass(a, geographic_, iscale_, nsplit, qdiag_.get(), stream_), "hat pass");
    stats_.kernel_launches += nsplit > 1 ? 1 : 0;
}

void Engine::hatAll(double bw, bool adaptive, int kernel, const double* ainv, double* S0, double* SA)
{
    check(cudaSetDevice(device_), "cudaSetDevice");
    computeThresholds(bw, adaptive);
    check(launch_mgwr_hat_all(points(), geographic_, x_.get(), p_, ainv, thrPtr(adaptive), bw, kernel, S0, SA,
                              num_sms_, stream_),
          "hat all");
    stats_.kernel_launches += 1;
}

void Engine::hatUpdate(double bw, bool adaptive, int kernel, const double* T, double* SA)
{
    if (p_ != 1) throw std::logic_error("hatUpdate needs the one-variable problem");
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int saved = precision_;
    precision_ = kFP64;
    struct Restore {
        int& slot;
        int value;
        ~Restore() { slot = value; }
    } restore{precision_, saved};
    computeThresholds(bw, adaptive);
    const int* unless = hatUpdateFx(bw, adaptive, kernel, T, SA) ? hat_state_.get() : nullptr;
    check(launch_mgwr_hat_update(points(), geographic_, tb16_.get(), x_.get(), vvec_.get(), thrPtr(adaptive), bw,
                                 kernel, T, SA, unless, stream_),
          "hat update");
    stats_.kernel_launches += 1;
}

// SA = S (T + I) by the fixed-point contraction: its columns are the n columns of
// x_j (T + I), 64 at a time, where the FP64 kernel needs n FMAs a pair.  False when
// it does not apply (kernel, coordinates) or its digit images (16 bytes a value) do
// not fit beside the matrices; otherwise the FP64 kernel runs only if hat_state_
// tells that T is not finite.
bool Engine::hatUpdateFx(double bw, bool adaptive, int kernel, const double* T, double* SA)
{
    // v_i is as large as the variable's weights near i are small, if x_i is not 0 (then the
    // row is 0): weights below 2^-62 would be missing from s_ij = v_i w_ij x_j up to 2^-32
    if (!fxReady(bw, adaptive, kernel) || !ixy_exact_ || (guard_hit_ & 2)) return false;
    const int tiles = (n_ + kTile - 1) / kTile, groups = (n_ + 63) / 64;
    const size_t bytes = (size_t)tiles * groups * 64 * 256;
    if (!fx_fits(64, tiles)) return false;
    if (hat_img_.capacityBytes() < bytes) {
        size_t free_b = 0, total_b = 0;
        check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
        const auto fits = [&] { return bytes + (bytes >> 3) + (1u << 30) <= free_b; };
        if (!fits() && release_idle_scratch()) check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
        if (!fits()) return false;
        hat_img_.alloc(bytes);
    }
    hat_exp_.alloc((size_t)((n_ + 1023) / 1024) * groups * 64);
    hat_state_.alloc(1);
    check(launch_build_zfx(n_, n_, 64, groups, T, n_, x_.get(), hat_img_.get(), hat_exp_.get(), nullptr,
                           hat_state_.get(), stream_),
          "build_zfx");
    FxArgs a = fxArgs(bw, adaptive ? thr_.get() : nullptr);
    setFocus(a, fxFocus(), tb16_.get(), n_, true);
    a.wpow = 1;
    a.ncols = n_;
    a.N = 64;
    a.zgroups = groups;
    a.zimg = hat_img_.get();
    a.zexp = hat_exp_.get();
    a.zcols = groups * 64;
    a.out = SA;
    a.ldo = n_;
    a.rowscale = vvec_.get();
    fx_rowmax_.alloc(n_);
    a.rowmax = fx_rowmax_.get();
    check(launch_contract_fx(a, fxMode(kernel), 1, stream_), "contract_fx");
    stats_.kernel_launches += 2;
    return true;
}

void Engine::synchronizeFx()
{
    if (zfx_ready_)
        check(cudaMemcpyAsync(host_sums_ + 6, fx_state_.get(), 3 * sizeof(int), cudaMemcpyDeviceToHost, stream_), "D2H");
    synchronize();
    if (zfx_ready_) fxCheck();
}

void Engine::releaseHatScratch()
{
    hat_img_.release();
    hat_exp_.release();
}

void Engine::copyOut(const double* dev, int cols, std::vector<double>& out)
{
    out_.alloc((size_t)n_ * cols);
    UnpermuteArgs u{};
    u.n = n_;
    u.perm = d_perm_.get();
    u.p[0] = cols;
    u.src[0] = dev;
    u.dst[0] = out_.get();
    check(launch_unpermute(u, 1, stream_), "unpermute");
    out.resize((size_t)n_ * cols);
    check(cudaMemcpyAsync(out.data(), out_.get(), sizeof(double) * out.size(), cudaMemcpyDeviceToHost, stream_), "D2H");
    synchronize();
}

void Engine::betas(std::vector<double>& out) { copyOut(beta_.get(), p_, out); }
void Engine::betasSE(std::vector<double>& out) { copyOut(bse_.get(), p_, out); }

// FP32 proxy coordinates and 32-point tile bounds shared by the select and the
// mixed path.
void Engine::buildProxy()
{
    const int n = n_, p = p_;
    ntiles32_ = (n + 31) / 32;
    boxes32_.alloc(ntiles32_);
    // planar frame of the FP32 records and bounds: the centroid, and a slack of
    // a few ulp of the largest relative coordinate
    uc_ = vc_ = 0.0;
    double maxabs = 0.0;
    if (!geographic_) {
        for (int s = 0; s < n; s++) {
            uc_ += hu_[s];
            vc_ += hv_[s];
        }
        uc_ /= n;
        vc_ /= n;
        for (int s = 0; s < n; s++) maxabs = std::max(maxabs, std::max(std::fabs(hu_[s] - uc_), std::fabs(hv_[s] - vc_)));
    }
    slack_ = std::ldexp(maxabs, -20);
    const int nt16 = (n + kTile - 1) / kTile, nt1024 = (n + 1023) / 1024;
    rvec_.alloc((size_t)n * p);
    pts32_.alloc((size_t)ntiles32_ * 32 * (geographic_ ? 2 : 1));
    tbsel_.alloc(ntiles32_);
    tb16_.alloc(nt16);
    stb_.alloc(nt1024);
    if (!geographic_) {
        caps32_.clear();
        check(launch_planar_proxy(n, u_.get(), v_.get(), uc_, vc_, slack_, tiles_.get(), boxes32_.get(), tb16_.get(),
                                  tbsel_.get(), stb_.get(), pts32_.get(), stream_),
              "planar records and bounds");
        stats_.kernel_launches += 1;
    } else {
        const std::vector<float4> pts = point_records(he_);
        const std::vector<TileCap> c32 = make_caps(he_, 32);
        const std::vector<TileBox> bx = make_boxes(hu_, hv_, 32);
        const std::vector<float4> tb = tile_bounds(he_, 32);
        const std::vector<float4> t16 = tile_bounds(he_, kTile);
        const std::vector<float4> t1024 = tile_bounds(he_, 1024);
        caps32_.alloc(c32.size());
        auto up = [&](void* dst, const void* src, size_t bytes) {
            check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream_), "H2D tile bounds");
        };
        up(caps32_.get(), c32.data(), sizeof(TileCap) * c32.size());
        up(boxes32_.get(), bx.data(), sizeof(TileBox) * bx.size());
        up(pts32_.get(), pts.data(), sizeof(float4) * pts.size());
        up(tbsel_.get(), tb.data(), sizeof(float4) * tb.size());
        up(tb16_.get(), t16.data(), sizeof(float4) * t16.size());
        up(stb_.get(), t1024.data(), sizeof(float4) * t1024.size());
        synchronize();
    }
    // proxy error bands of the exact select.  The FP32 great-circle proxy is within
    // 5.3e-7 relative of the reference's distance wherever it is trusted (d < 15,000 km;
    // measured over near, regional and global pairs), 1e-10 km absolute for nearly
    // coincident points: 2^-16 (1.5e-5) and 1e-6 km leave a margin of 25x over it.
    // Every point inside the band is evaluated with the correctly rounded formula.
    if (!geographic_) {
        sel_eps_ = std::ldexp(1.0, -18);
        sel_delta_ = std::ldexp(dhi_, -36);
    } else {
        sel_eps_ = std::ldexp(1.0, -16);
        sel_delta_ = 1e-6;
    }
    tile_thr16_.alloc(nt16);
    sel_err_.alloc(1);
    check(cudaMemsetAsync(sel_err_.get(), 0, sizeof(int), stream_), "memset");
    synchronize();
}

// Mixed-precision operands: X and y centred (when a constant column is the
// intercept) and scaled, Z~ split into TF32 hi/lo swizzled tile images, FP32
// hi/lo coordinates, 32-point tile boxes.
void Engine::ensureMixed()
{
    if (mixed_ready_) return;
    const int n = n_, p = p_;
    if (m_ > 256) throw std::invalid_argument("mixed precision supports at most 21 columns of X");
    npad_ = (m_ + 15) / 16 * 16;  // the accumulator width: the tcgen05 N of an M = 128 MMA is a multiple of 16
    xs_.alloc((size_t)n * p);
    ys_.alloc(n);
    zs_.alloc((size_t)n * m_);
    zimg_.alloc((size_t)ntiles32_ * 2 * npad_ * 128);
    acc_.alloc((size_t)(n + 127) / 128 * 128 * npad_);  // rows in groups of 128 (the contraction's layout)
    stage_.alloc((size_t)(n + 127) / 128 * 128 * npad_);
    thr32_.alloc(n);
    err_.alloc(1);
    tinv_.alloc(p);
    tvec_.alloc(p);
    musc_.alloc(2 * p + 3);
    prep_.alloc(column_stats_bytes(n, p));
    check(launch_column_stats(n, p, x_.get(), y_.get(), prep_.get(), musc_.get(), tinv_.get(), tvec_.get(), xs_.get(),
                              ys_.get(), stream_),
          "column statistics");
    stats_.kernel_launches += 5;
    double of_y[3];
    check(cudaMemcpyAsync(of_y, musc_.get() + 2 * p, sizeof(of_y), cudaMemcpyDeviceToHost, stream_), "D2H");
    check(cudaMemsetAsync(err_.get(), 0, sizeof(int), stream_), "memset err");
    check(launch_build_z(n, p, xs_.get(), ys_.get(), zs_.get(), stream_), "build_z");
    check(launch_build_zimg(n, m_, npad_, zs_.get(), m_, zimg_.get(), stream_), "build_zimg");
    synchronize();
    mu_y_ = of_y[0];
    s_y_ = of_y[1];
    intercept_col_ = (int)of_y[2];
    mixed_ready_ = true;
}

cudaEvent_t Engine::timerBegin()
{
    cudaEvent_t e0 = nullptr;
    check(cudaEventCreate(&e0), "event");
    check(cudaEventRecord(e0, stream_), "event record");
    return e0;
}

void Engine::timerEnd(cudaEvent_t e0, int kind)
{
    cudaEvent_t e1 = nullptr;
    check(cudaEventCreate(&e1), "event");
    check(cudaEventRecord(e1, stream_), "event record");
    pending_.push_back(PendingTiming{e0, e1, kind});
}

EngineStats& Engine::stats()
{
    for (auto& pt : pending_) {
        float ms = 0.f;
        if (cudaEventSynchronize(pt.e1) == cudaSuccess && cudaEventElapsedTime(&ms, pt.e0, pt.e1) == cudaSuccess)
            (pt.kind == 0 ? stats_.contract_ms : pt.kind == 1 ? stats_.select_ms : stats_.d2c_fill_ms) += ms;
        cudaEventDestroy(pt.e0);
        cudaEventDestroy(pt.e1);
    }
    pending_.clear();
    if (counters_dirty_ && tile_count_.get()) {
        unsigned long long tiles = 0, pc[kTcProfSlots];
        check(cudaMemcpyAsync(&tiles, tile_count_.get(), sizeof(tiles), cudaMemcpyDeviceToHost, stream_), "D2H");
        check(cudaMemcpyAsync(pc, tc_prof_.get(), sizeof(pc), cudaMemcpyDeviceToHost, stream_), "D2H");
        check(cudaMemsetAsync(tile_count_.get(), 0, sizeof(unsigned long long), stream_), "memset tiles");
        check(cudaMemsetAsync(tc_prof_.get(), 0, sizeof(pc), stream_), "memset prof");
        synchronize();
        stats_.contract_tiles += (long long)tiles;
        for (int q = 0; q < kTcProfSlots && q < 12; q++) {
            if (q == kTcProfLoopMax || q == kTcProfTilesMax)
                stats_.contract_phase_cycles[q] = std::max(stats_.contract_phase_cycles[q], (double)pc[q]);
            else
                stats_.contract_phase_cycles[q] += (double)pc[q];
        }
        counters_dirty_ = false;
    }
    return stats_;
}

void Engine::resetStats()
{
    stats();
    stats_ = EngineStats{};
}

void Engine::contractMixed(double* G, int ldg, int mcols, double bw, bool adaptive, int kernel, bool exclude_self,
                           int wpow)
{
    if (adaptive) {
        check(launch_to_float(n_, thr_.get(), thr32_.get(), stream_), "thr32");
        stats_.kernel_launches += 1;
    }
    TcArgs a{};
    a.n = n_;
    a.mcols = mcols;
    a.npad = npad_;
    a.ntiles = ntiles32_;
    a.pts = pts32_.get();
    a.tb = tbsel_.get();
    a.zimg = zimg_.get();
    a.thr = adaptive ? thr32_.get() : nullptr;
    a.bw = (float)bw;
    a.kernel = kernel;
    a.exclude_self = exclude_self ? 1 : 0;
    a.skip = 1;
    a.flush_tiles = flush_tiles_;
    a.wait_limit = tc_wait_limit_;
    a.wpow = wpow;
    const size_t acc_size = (size_t)(n_ + 127) / 128 * 128 * npad_;
    // the tiles a row block visits: all of them, about twice those that hold the neighbours,
    // or (a fixed bandwidth and a compact kernel) any number: no split
    const bool compact = adaptive && kernel >= GW_KERNEL_BISQUARE;
    // (in whole chunks: an estimate of the engine's memory goes through every number)
    int visits = compact ? (int)std::min((double)ntiles32_, bw / 16 + 8) : ntiles32_;
    visits = std::min(ntiles32_, (visits + flush_tiles_ - 1) / flush_tiles_ * flush_tiles_);
    // (the splits group the sums: their number follows from the shape, and from the memory
    // only where the call would fail for want of it)
    a.nsplit = !adaptive && kernel >= GW_KERNEL_BISQUARE ? 1 : tc_splits((n_ + 127) / 128, visits, flush_tiles_, num_sms_);
    if (!acc_.tryAlloc(a.nsplit * acc_size) || !stage_.tryAlloc(a.nsplit * acc_size)) {
        a.nsplit = 1;
        acc_.release();
        acc_.alloc(acc_size);
        stage_.alloc(acc_size);
    }
    a.acc_stride = acc_size;
    a.acc = acc_.get();
    a.stage = stage_.get();
    a.G = G;
    a.ldg = ldg;
    a.err = err_.get();
    // geographic: the pair distances come from the device's distance cache when it fits
    DeviceD2Cache& dc = device_d2c(device_);
    std::unique_lock<std::mutex> d2lock(dc.mu, std::defer_lock);
    if (geographic_ && d2c_limit_bytes_ != 0) {
        d2lock.lock();
        a.d2c = ensureDistanceCache();
        if (!a.d2c) d2lock.unlock();
    }
    cudaEvent_t e0 = stats_on_ ? timerBegin() : nullptr;
    if (stats_on_) {
        if (!tile_count_.get()) {
            tile_count_.alloc(1);
            tc_prof_.alloc(kTcProfSlots);
            check(cudaMemsetAsync(tile_count_.get(), 0, sizeof(unsigned long long), stream_), "memset tiles");
            check(cudaMemsetAsync(tc_prof_.get(), 0, sizeof(unsigned long long) * kTcProfSlots, stream_),
                  "memset prof");
        }
        a.tiles = tile_count_.get();
        a.prof = phases_on_ ? tc_prof_.get() : nullptr;
        counters_dirty_ = true;
    }
    check(launch_contract_tc(a, geographic_, stream_), "contract_tc");
    stats_.kernel_launches += a.nsplit > 1 ? 2 : 1;
    if (a.d2c) {
        check(cudaEventRecord(dc.used, stream_), "cudaEventRecord");
        d2lock.unlock();
    }
    if (stats_on_) {
        timerEnd(e0, 0);
        stats_.contract_launches += 1;
        double pairs = (double)n_ * n_;
        if (adaptive && kernel >= GW_KERNEL_BISQUARE) pairs = (double)n_ * std::max(0.0, std::min(bw, (double)n_) - 1);
        stats_.contract_flops += 2.0 * mcols * pairs;
        stats_.contract_bytes += 2.0 * npad_ * 128.0 * ntiles32_ * 2 + 8.0 * n_ * mcols + 16.0 * n_;
        if (a.d2c) stats_.contract_bytes += 4.0 * pairs;  // the cached distances of the nonzero pairs
    }
}

void Engine::tcSelftest(int N, const float* A, const float* B, float* D)
{
    check(cudaSetDevice(device_), "cudaSetDevice");
    DevBuf<float> dA, dB, dD;
    DevBuf<int> derr;
    dA.alloc(128 * 32);
    dB.alloc((size_t)N * 32);
    dD.alloc((size_t)128 * N);
    derr.alloc(1);
    check(cudaMemcpyAsync(dA.get(), A, sizeof(float) * 128 * 32, cudaMemcpyHostToDevice, stream_), "H2D");
    check(cudaMemcpyAsync(dB.get(), B, sizeof(float) * N * 32, cudaMemcpyHostToDevice, stream_), "H2D");
    check(cudaMemsetAsync(derr.get(), 0, sizeof(int), stream_), "memset");
    check(launch_tc_selftest(dA.get(), dB.get(), dD.get(), N, derr.get(), stream_), "tc selftest");
    int err = 0;
    check(cudaMemcpyAsync(D, dD.get(), sizeof(float) * 128 * N, cudaMemcpyDeviceToHost, stream_), "D2H");
    check(cudaMemcpyAsync(&err, derr.get(), sizeof(int), cudaMemcpyDeviceToHost, stream_), "D2H");
    synchronize();
    if (err) throw CudaError("tensor-core self-test: a bounded wait timed out");
}

// Per-row order statistic of the given rank (1-based), computed once and kept
// for the dataset.  The first select also stores every row's histogram of
// proxy distances, so later ranks start from the right histogram bin.
const double* Engine::orderStatistic(unsigned rank)
{
    const bool exact = precision_ == kFP64;
    for (auto& e : ranks_)
        if (e->exact == exact && e->rank == rank) return e->v.get();
    if (ranks_.size() >= 64) recycleRanks();
    if (!hist_tried_) {
        hist_tried_ = true;
        const size_t bytes = (size_t)n_ * (4096 + 64) * sizeof(unsigned);
        bool fits;
        if (hist_limit_bytes_ >= 0) {
            fits = bytes <= (size_t)hist_limit_bytes_;
        } else {
            size_t free_b = 0, total_b = 0;
            cudaMemGetInfo(&free_b, &total_b);
            fits = bytes < free_b / 4 || bytes <= hist_.capacityBytes() + hcoarse_.capacityBytes();
            if (!fits && release_idle_scratch()) {
                cudaMemGetInfo(&free_b, &total_b);
                fits = bytes < free_b / 4;
            }
        }
        if (fits) {
            hist_.alloc((size_t)n_ * 4096);
            hcoarse_.alloc((size_t)n_ * 64);
        }
        hist_valid_ = false;
    }
    std::unique_ptr<RankStat> r;
    if (!rank_pool_.empty()) {
        r = std::move(rank_pool_.back());
        rank_pool_.pop_back();
    } else {
        r.reset(new RankStat);
    }
    r->rank = rank;
    r->exact = exact;
    r->v.alloc(n_);
    SelectArgs a{};
    a.n = n_;
    a.ntiles = ntiles32_;
    a.P = points();
    a.pts = pts32_.get();
    a.tb = tbsel_.get();
    a.stb = stb_.get();
    a.hist_cache = hist_.get();
    a.cache_valid = hist_valid_ ? 1 : 0;
    a.hist_coarse = hist_.get() ? hcoarse_.get() : nullptr;
    a.rank = rank;
    a.dlo = dlo_;
    a.dhi = dhi_;
    a.eps = sel_eps_;
    a.delta = sel_delta_;
    a.out = r->v.get();
    a.err = sel_err_.get();
    if (hist_.get() && !hist_valid_) {
        // geographic mixed data: the distance cache is filled first (each pair once,
        // the distance being symmetric) and the histograms are read back from it
        DeviceD2Cache& dc = device_d2c(device_);
        std::unique_lock<std::mutex> lk(dc.mu, std::defer_lock);
        const float* cache = nullptr;
        if (geographic_ && precision_ == kMixed && d2c_limit_bytes_ != 0) {
            lk.lock();
            cache = ensureDistanceCache();
            if (!cache) lk.unlock();
        }
        if (cache) {
            a.d2c = cache;
            check(launch_select_hist_cached(a, num_sms_, stream_), "select histograms");
            a.d2c = nullptr;
            check(cudaEventRecord(dc.used, stream_), "cudaEventRecord");
            lk.unlock();
        } else {
            check(launch_select_hist(a, geographic_, num_sms_, stream_), "select histograms");
        }
        stats_.kernel_launches += 1;
        hist_valid_ = true;
        a.cache_valid = 1;
    }
    // geographic mixed data whose distance cache is filled: the select reads the
    // histogram pass's proxy values from it instead of recomputing them
    DeviceD2Cache& dc = device_d2c(device_);
    std::unique_lock<std::mutex> lk(dc.mu, std::defer_lock);
    if (geographic_ && precision_ == kMixed && d2c_valid_) {
        lk.lock();
        if (dc.owner == this && d2c_valid_ && dc.ptr) a.d2c = dc.ptr;
        else lk.unlock();
    }
    if (geographic_ && exact) {
        sel_defer_.alloc(n_);
        a.defer = sel_defer_.get();
        stats_.kernel_launches += 1;
    }
    check(launch_select(a, geographic_, exact, num_sms_, stream_), "select");
    stats_.kernel_launches += 1;
    if (a.d2c) {
        check(cudaEventRecord(dc.used, stream_), "cudaEventRecord");
        lk.unlock();
    }
    if (hist_.get()) hist_valid_ = true;
    ranks_.push_back(std::move(r));
    return ranks_.back()->v.get();
}

void Engine::computeThresholds(double bw, bool adaptive)
{
    if (!adaptive) return;
    if (thr_valid_ && thr_bw_ == bw && thr_prec_ == precision_) return;
    const double dn = bw / n_;
    cudaEvent_t e0 = stats_on_ ? timerBegin() : nullptr;
    if (dn < 1) {
        // d0 = vdist(int(b0) - 1), d1 = vdist(int(b0)) (BandwidthWeight.cpp:46-48)
        const double b0 = std::floor(bw), bx = bw - b0;
        const long long r0 = (long long)(int)b0;
        if (r0 < 1 || r0 >= n_) throw std::out_of_range("Mat::operator(): index out of bounds");
        const double* d0 = orderStatistic((unsigned)r0);
        const double* d1 = bx != 0.0 ? orderStatistic((unsigned)(r0 + 1)) : nullptr;
        check(launch_threshold_combine(n_, bw, d0, d1, thr_.get(), stream_), "threshold");
    stats_.kernel_launches += 1;
    } else {
        // fixbw = dn * max(dist) (BandwidthWeight.cpp:50-53)
        const double* dmax = orderStatistic((unsigned)n_);
        check(launch_threshold_combine(n_, bw, dmax, nullptr, thr_.get(), stream_), "threshold");
    stats_.kernel_launches += 1;
    }
    if (stats_on_) {
        timerEnd(e0, 1);
        stats_.select_launches += 1;
    }
    thr_valid_ = true;
    thr_bw_ = bw;
    thr_prec_ = precision_;
}

// Integer coordinates of n points on the device; false when one does not fit, exact
// cleared when a bit was lost.
bool Engine::integerCoords(int n, const double* u, const double* v, DevBuf<longlong2>& out, bool& exact)
{
    out.alloc(n);
    prep_flags_.alloc(2);
    check(launch_int_coords(n, u, v, iu0_, iv0_, iscale_, out.get(), prep_flags_.get(), stream_), "integer coordinates");
    stats_.kernel_launches += 1;
    int f[2];
    check(cudaMemcpyAsync(f, prep_flags_.get(), sizeof(f), cudaMemcpyDeviceToHost, stream_), "D2H");
    synchronize();
    if (f[1]) exact = false;
    return f[0] == 0;
}

// Whether points with these unit vectors (3 x n) and the data, whose cap is centred
// at ec_, lie within one spherical cap of chord radius 1/2: every haversine is then
// below 1/4.
bool Engine::withinCap(const std::vector<double>& e) const
{
    const size_t n = e.size() / 3;
    for (size_t i = 0; i < n; i++) {
        const double dx = e[i] - ec_[0], dy = e[n + i] - ec_[1], dz = e[2 * n + i] - ec_[2];
        const double d = dx * dx + dy * dy + dz * dz;
        if (!(d < 0.2499)) return false;
    }
    return true;
}

// Whether the fixed-point contraction applies to the resident data and kernel;
// builds its operands on first use.  Bisquare and gaussian weights are functions
// of the squared distance alone; the other kernels keep the FP64 form, and so do
// great-circle distances of data wider than a cap of 3,200 km radius, where the
// polynomials of fx_geo.cuh end.
bool Engine::fxReady(double bw, bool adaptive, int kernel)
{
    if (kernel != GW_KERNEL_BISQUARE && kernel != GW_KERNEL_GAUSSIAN) return false;
    // fixed-point rows need a positive finite threshold (an infinite one weighs every pair 1)
    if (!adaptive && !(bw > 0.0 && std::isfinite(bw))) return false;
    if (zfx_ready_ && zfx_kind_ == 1 && zfx_bad_ == 1) return false;
    const int tiles = (n_ + kTile - 1) / kTile;
    int groups = 0;
    const int N = fx_columns(m_, &groups);
    if (!fx_fits(N, tiles)) return false;
    if (!ixy_tried_ && geographic_) {
        ixy_tried_ = true;
        double c[3] = {0.0, 0.0, 0.0};
        for (int q = 0; q < 3; q++)
            for (int i = 0; i < n_; i++) c[q] += he_[(size_t)q * n_ + i];
        const double nrm = std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
        for (int q = 0; q < 3; q++) ec_[q] = c[q] / nrm;
        ixy_ok_ = ixy_exact_ = nrm > 0.0 && withinCap(he_);
        if (ixy_ok_) {
            ie3_.alloc(n_);
            check(launch_int_vectors(n_, uR_.get(), vR_.get(), ie3_.get(), stream_), "integer unit vectors");
            stats_.kernel_launches += 1;
            if (!geo_.get()) {
                std::vector<fx::GeoCoef> g(fx::kGeoIntervals);
                fx::geo_table(g.data());
                geo_.alloc(g.size());
                check(cudaMemcpyAsync(geo_.get(), g.data(), sizeof(fx::GeoCoef) * g.size(), cudaMemcpyHostToDevice,
                                      stream_),
                      "H2D polynomials");
                synchronize();  // g goes away
            }
        }
    }
    if (!ixy_tried_) {
        ixy_tried_ = true;
        double umin = hu_[0], umax = umin, vmin = hv_[0], vmax = vmin;
        for (int i = 0; i < n_; i++) {
            umin = std::min(umin, hu_[i]);
            umax = std::max(umax, hu_[i]);
            vmin = std::min(vmin, hv_[i]);
            vmax = std::max(vmax, hv_[i]);
        }
        const double extent = std::max(umax - umin, vmax - vmin);
        ixy_ok_ = std::isfinite(extent) && (extent == 0.0 || (extent > 1e-250 && extent < 1e250));
        if (ixy_ok_) {
            iscale_ = extent > 0.0 ? 60 - std::ilogb(extent) : 0;
            iu0_ = umin;
            iv0_ = vmin;
            ixy_exact_ = true;
            ixy_ok_ = integerCoords(n_, u_.get(), v_.get(), ixy_, ixy_exact_);
        }
    }
    if (!ixy_ok_) return false;
    if (!zfx_ready_ || zfx_kind_ != 1) buildZfx(false);
    return true;
}

bool Engine::buildZfx(bool mixed)
{
    const int tiles = (n_ + kTile - 1) / kTile;
    zfx_n_ = fx_columns(m_, &zfx_groups_);
    zfx_.alloc((size_t)tiles * zfx_groups_ * zfx_n_ * 256);
    const size_t scales = (size_t)((n_ + 1023) / 1024) * zfx_groups_ * zfx_n_;
    zfx_exp_.alloc(scales);
    zfx_sum_.alloc(2 * scales);
    fx_lim_.alloc(2 * (size_t)p_);
    if (!fx_state_.get()) {
        fx_state_.alloc(3);
        check(cudaMemsetAsync(fx_state_.get(), 0, 3 * sizeof(int), stream_), "memset");
    }
    check(launch_build_zfx(n_, m_, zfx_n_, zfx_groups_, mixed ? zs_.get() : z_.get(), m_, nullptr, zfx_.get(),
                           zfx_exp_.get(), zfx_sum_.get(), fx_state_.get(), stream_),
          "build_zfx");
    stats_.kernel_launches += 1;
    zfx_ready_ = true;
    zfx_kind_ = mixed ? 2 : 1;
    zfx_bad_ = -1;
    if (mixed) {  // the caller has no FP64 sums to fall back on in the same stream: ask now, once per X and y
        check(cudaMemcpyAsync(host_sums_ + 6, fx_state_.get(), 3 * sizeof(int), cudaMemcpyDeviceToHost, stream_), "D2H");
        synchronize();
        fxCheck();
    }
    return zfx_bad_ != 1;
}

// The residuals of the refinement as b - A beta, with A and b the exact sums of the
// contraction's FP32 weights (the fixed-point contraction over their digits) in
// place of a double-float pass over every pair, p times as long.  False when the
// digit images do not apply.
bool Engine::refineFx(double bw, bool adaptive, int kernel, const float* d2c)
{
    const int tiles = (n_ + kTile - 1) / kTile;
    int groups = 0;
    if (!fx_fits(fx_columns(m_, &groups), tiles)) return false;
    if (zfx_ready_ && zfx_kind_ == 2 ? zfx_bad_ == 1 : !buildZfx(true)) return false;
    FxArgs a{};
    a.n = a.nf = n_;
    a.ntiles = tiles;
    a.pts = a.fpts = pts32_.get();
    a.thr32 = adaptive ? thr32_.get() : nullptr;
    a.bw = bw;
    a.kernel = kernel;
    a.d2c = d2c;
    a.tb16 = a.ftb16 = tb16_.get();
    a.wpow = 1;
    a.ncols = m_;
    a.N = zfx_n_;
    a.zgroups = zfx_groups_;
    a.zimg = zfx_.get();
    a.zexp = zfx_exp_.get();
    a.zcols = zfx_n_ * zfx_groups_;
    a.err = fx_state_.get() + 1;
    a.wait_limit = tc_wait_limit_;
    a.limits = fxLimits(bw, adaptive, kernel, 1);
    // the contraction's sums are free by now: rows of at most npad doubles
    double* G = reinterpret_cast<double*>(acc_.get());
    const int nsplit = fx_splits((n_ + 127) / 128 * zfx_groups_, tiles, num_sms_);
    fx_rowmax_.alloc((size_t)nsplit * n_);
    a.rowmax = fx_rowmax_.get();
    a.ldo = m_;
    a.out = G;
    if (nsplit > 1) {
        a.split_stride = (size_t)n_ * m_;
        fx_part_.alloc(a.split_stride * nsplit);
        a.out = fx_part_.get();
    }
    check(launch_contract_fx(a, geographic_ ? kFxMixedGeo : kFxMixed, nsplit, stream_), "contract_fx");
    check(launch_fx_finish(a, nsplit, G, m_, nullptr, stream_), "fx_finish");
    refine_low_.alloc((n_ + kResidualRows - 1) / kResidualRows);
    check(launch_normal_residual(n_, p_, G, m_, beta_.get(), fx_lim_.get(), rvec_.get(), refine_low_.get(), stream_),
          "residual");
    stats_.kernel_launches += nsplit > 1 ? 3 : 2;
    return true;
}

FxMode Engine::fxMode(int kernel) const
{
    const bool gauss = kernel == GW_KERNEL_GAUSSIAN;
    return geographic_ ? (gauss ? kFxGeoGauss : kFxGeoBisquare) : (gauss ? kFxGauss : kFxBisquare);
}

// The data side of the fixed-point contraction.
FxArgs Engine::fxArgs(double bw, const double* thr) const
{
    FxArgs a{};
    a.n = n_;
    a.ntiles = (n_ + kTile - 1) / kTile;
    if (geographic_) {
        a.pe3 = ie3_.get();
        a.geo = geo_.get();
    } else {
        a.pxy = ixy_.get();
    }
    a.scale = iscale_;
    a.tb16 = tb16_.get();
    a.thr = thr;
    a.bw = bw;
    a.err = fx_state_.get() + 1;
    a.wait_limit = tc_wait_limit_;
    return a;
}

// Its focus rows: integer coordinates or unit vectors, as the data's.
void Engine::setFocus(FxArgs& a, const void* focus, const float4* ftb16, int nf, bool exact) const
{
    if (geographic_) a.fe3 = (const fx::Vec3*)focus;
    else a.fxy = (const longlong2*)focus;
    a.ftb16 = ftb16;
    a.nf = nf;
    a.exact = exact ? 1 : 0;
}

// The device's buffer for kept weights (bytes), or null where it may not grow to that size.
// Waits for an engine that is between its passes: on the host for the launches of the
// other passes, on the stream for their end.
unsigned long long* Engine::takeWeights(size_t bytes)
{
    if (bytes > (size_t)scratch_limit_bytes_) return nullptr;
    DeviceWeights& w = g_weights[device_];
    std::unique_lock<std::mutex> lk(w.mu);
    w.idle.wait(lk, [&] { return !w.user || w.user == this; });
    if (w.bytes < bytes) {
        free_weights(w);
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || bytes >= free_b / 8 ||
            cudaMalloc(&w.ptr, bytes) != cudaSuccess) {
            cudaGetLastError();
            w.ptr = nullptr;
            return nullptr;
        }
        w.bytes = bytes;
    }
    if (!w.used) check(cudaEventCreateWithFlags(&w.used, cudaEventDisableTiming), "cudaEventCreate");
    check(cudaStreamWaitEvent(stream_, w.used, 0), "cudaStreamWaitEvent");
    w.user = this;
    return w.ptr;
}

void Engine::leaveWeights()
{
    DeviceWeights& w = g_weights[device_];
    std::lock_guard<std::mutex> lk(w.mu);
    fx_weights_kept_ = false;
    if (w.user != this) return;
    cudaEventRecord(w.used, stream_);
    w.user = nullptr;
    w.idle.notify_all();
}

// G over the first mcols columns of Z by the fixed-point contraction, for the
// focus rows given as integer coordinates and tile bounds.  Returns whether
// fx_flags_ now marks row blocks for k_contract64: rows that exclude their own
// weight or are not data points may have small weights only, and rounded
// coordinates may be too coarse for a small threshold; every other row holds its
// own weight 1.  Until the first synchronisation has told whether Z suits, the
// FP64 kernel is launched behind it too (it leaves at once when it does).
bool Engine::contractFx(const void* focus, const float4* ftb16, int nf, int mcols, double* G, int ldg,
                        const double* thr, double bw, int kernel, bool exclude_self, int wpow, bool exact,
                        const FxLimits& limits, WeightUse use)
{
    const bool flags = exclude_self || focus != fxFocus() || !exact || zfx_bad_ < 0;
    FxArgs a = fxArgs(bw, thr);
    setFocus(a, focus, ftb16, nf, exact);
    a.exclude_self = exclude_self ? 1 : 0;
    a.wpow = wpow;
    a.ncols = mcols;
    a.N = zfx_n_;
    a.zgroups = zfx_groups_;
    a.zimg = zfx_.get();
    a.zexp = zfx_exp_.get();
    a.zcols = zfx_n_ * zfx_groups_;
    a.limits = limits;
    const int groups = (mcols + zfx_n_ - 1) / zfx_n_;
    // Further column groups and passes read the first group's weights back: making them
    // takes some 10 times as long as the rest of a tile (n = 20,011, p = 17, great-circle).
    const bool load = use == WeightUse::kAgain && fx_weights_kept_;
    const bool wanted = load || groups > 1 || use == WeightUse::kKept;
    unsigned long long* const weights = wanted ? takeWeights(fx_weight_bytes(nf, n_)) : nullptr;
    const bool store = weights && !load;
    if (use == WeightUse::kKept) fx_weights_kept_ = store;
    // (the splits group the sums: the same number whether or not the weights fit)
    const int nsplit = fx_splits((nf + 127) / 128 * (use == WeightUse::kAgain ? groups : 1), a.ntiles, num_sms_);
    fx_rowmax_.alloc((size_t)nsplit * nf);
    a.rowmax = fx_rowmax_.get();
    if (nsplit > 1) {
        a.ldo = mcols;
        a.split_stride = (size_t)nf * mcols;
        fx_part_.alloc(a.split_stride * nsplit);
        a.out = fx_part_.get();
    } else {
        a.out = G;
        a.ldo = ldg;
    }
    if (flags) fx_flags_.alloc((nf + kRowBlock - 1) / kRowBlock);
    if (load) a.wload = weights;
    if (store) {
        a.wstore = weights;
        a.groups = 1;
    }
    check(launch_contract_fx(a, fxMode(kernel), nsplit, stream_), "contract_fx");
    if (store && groups > 1) {
        a.wload = a.wstore;
        a.wstore = nullptr;
        a.group0 = 1;
        a.groups = groups - 1;
        check(launch_contract_fx(a, fxMode(kernel), nsplit, stream_), "contract_fx");
        stats_.kernel_launches += 1;
    }
    if (weights && !fx_weights_kept_) leaveWeights();
    check(launch_fx_finish(a, nsplit, G, ldg, flags ? fx_flags_.get() : nullptr, stream_), "fx_finish");
    stats_.kernel_launches += nsplit > 1 || flags ? 2 : 1;
    return flags;
}

void Engine::fxCheck()
{
    int st[3];
    std::memcpy(st, host_sums_ + 6, sizeof(st));
    zfx_bad_ = st[0] != 0;
    guard_hit_ |= st[2];
    if (st[1] || st[2]) {
        check(cudaMemsetAsync(fx_state_.get() + 1, 0, 2 * sizeof(int), stream_), "memset");
        synchronize();
    }
    if (st[1]) throw CudaError("fixed-point contraction: a bounded wait timed out");
}

FxLimits Engine::fxLimits(double bw, bool adaptive, int kernel, int wpow) const
{
    FxLimits l{};
    l.p = p_;
    // an adaptive threshold of a compact kernel leaves weight to the neighbours it counts
    l.points = adaptive && kernel >= GW_KERNEL_BISQUARE ? std::min((double)n_, bw + 1.0) : (double)n_;
    l.root = std::sqrt(l.points);
    l.zsum = zfx_sum_.get();
    l.off = fx_state_.get();
    l.lim = fx_lim_.get() + (wpow == 2 ? p_ : 0);
    return l;
}

FxGuard Engine::fxGuard(int rows, const int* done)
{
    const int blocks = (rows + kRowBlock - 1) / kRowBlock;
    if (guard_hit_ || (int)guard_flags_.size() != blocks) {  // otherwise no block is marked
        guard_flags_.alloc(blocks);
        check(cudaMemsetAsync(guard_flags_.get(), 0, sizeof(int) * blocks, stream_), "memset");
        guard_hit_ = 0;
    }
    FxGuard g{};
    g.lim = fx_lim_.get();
    g.done = done;
    g.flags = guard_flags_.get();
    g.any = fx_state_.get() + 2;
    return g;
}

// The blocks that guard_flags_ marks, for sums of up to mcols columns.
RowBlocks Engine::guardBlocks(int mcols)
{
    std::vector<int> marks(guard_flags_.size()), list;
    check(cudaMemcpyAsync(marks.data(), guard_flags_.get(), sizeof(int) * marks.size(), cudaMemcpyDeviceToHost, stream_),
          "D2H marks");
    synchronize();
    for (size_t b = 0; b < marks.size(); b++)
        if (marks[b]) list.push_back((int)b);
    guard_list_.alloc(list.size());
    check(cudaMemcpyAsync(guard_list_.get(), list.data(), sizeof(int) * list.size(), cudaMemcpyHostToDevice, stream_),
          "H2D blocks");
    synchronize();  // list goes away
    RowBlocks b{};
    b.list = guard_list_.get();
    b.count = (int)list.size();
    b.nsplit = contract64_splits(b.count, (n_ + kTile - 1) / kTile, num_sms_);
    if (b.nsplit > 1) fx_part_.alloc((size_t)b.nsplit * b.count * kRowBlock * std::min(256, mcols));
    b.part = fx_part_.get();
    return b;
}

// The FP64 contraction over every row block, or only some of them.
void Engine::contractRows(const double* Z, int mcols, double* G, int ldg, double bw, bool adaptive, int kernel,
                          bool exclude_self, int wpow, const RowBlocks& blocks)
{
    // the kernel takes at most 256 columns (p <= 21); wider Z (p up to 32) in column chunks
    for (int c0 = 0; c0 < mcols; c0 += 256) {
        const int w = std::min(256, mcols - c0);
        check(launch_contract64(points(), geographic_, tb16_.get(), Z + c0, m_, w, G + c0, ldg, thrPtr(adaptive), bw,
                                kernel, exclude_self, wpow, true, stream_, blocks),
              "contract64");
        stats_.kernel_launches += 1;
    }
}

void Engine::contract(const double* Z, int mcols, double* G, int ldg, double bw, bool adaptive, int kernel,
                      bool exclude_self, int wpow, WeightUse use)
{
    cudaEvent_t e0 = stats_on_ ? timerBegin() : nullptr;
    const bool fx = fxReady(bw, adaptive, kernel);
    const bool rest = !fx || contractFx(fxFocus(), tb16_.get(), n_, mcols, G, ldg, thrPtr(adaptive), bw, kernel,
                                        exclude_self, wpow, ixy_exact_,
                                        fxLimits(bw, adaptive, kernel, wpow), use);
    if (rest)
        contractRows(Z, mcols, G, ldg, bw, adaptive, kernel, exclude_self, wpow,
                     fx ? RowBlocks{fx_flags_.get(), fx_state_.get(), nullptr, 0, 0, nullptr} : RowBlocks{});
    if (wpow == 1) {
        g_fx_ = fx;
        g_flagged_ = fx && rest;
        g2_fx_ = false;
    } else {
        g2_fx_ = fx;
    }
    if (stats_on_) {
        timerEnd(e0, 0);
        stats_.contract_launches += 1;
        // useful pairs: dense kernels touch every pair; adaptive compact kernels
        // have b-1 neighbours with d < r_i per row (ties aside)
        double pairs = (double)n_ * n_;
        if (adaptive && kernel >= GW_KERNEL_BISQUARE) pairs = (double)n_ * std::max(0.0, std::min(bw, (double)n_) - 1);
        stats_.contract_flops += 2.0 * mcols * pairs;
        stats_.contract_bytes += 8.0 * ((double)n_ * m_ + (double)n_ * mcols) + 16.0 * n_;
    }
}

CriterionOut Engine::criterionOut()
{
    if (!ticket_.get()) {
        ticket_.alloc(1);
        check(cudaMemsetAsync(ticket_.get(), 0, sizeof(unsigned), stream_), "memset");
    }
    CriterionOut o{};
    o.host = host_sums_;
    o.sel_err = sel_err_.get();
    o.fx_state = zfx_ready_ ? fx_state_.get() : nullptr;
    o.ticket = ticket_.get();
    return o;
}

void Engine::solve(int mode, double bw, bool adaptive, int kernel, double out[4])
{
    SolveArgs a{};
    a.n = n_;
    a.p = p_;
    a.mode = mode;
    a.kernel = kernel;
    a.G = g_.get();
    a.ldg = m_;
    a.G2 = g2_.get();
    a.ldg2 = mm_;
    const bool mixed = precision_ == kMixed;
    a.X = mixed ? xs_.get() : x_.get();
    a.y = mixed ? ys_.get() : y_.get();
    a.thr = thrPtr(adaptive);
    a.bw = bw;
    // the criteria need no coefficients (the solve then skips the backward substitution)
    a.beta = (mode == kSolveAIC || mode == kSolveCV) ? nullptr : beta_.get();
    a.sii = sii_.get();
    a.resid = resid_.get();
    a.v = vvec_.get();
    a.bse = bse_.get();
    a.partials = partials_.get();
    a.tinv = mixed ? tinv_.get() : nullptr;
    a.tvec = (mixed && intercept_col_ >= 0) ? tvec_.get() : nullptr;
    a.tcol = mixed ? intercept_col_ : -1;
    a.rvec = rvec_.get();
    a.ainv = mode == kSolveFit ? ainv_out_ : nullptr;
    int nb = 0;
    const bool fx = zfx_ready_;
    a.out = criterionOut();
    if (mixed) a.out.err = err_.get();
    const bool guarded = !mixed && g_fx_ && zfx_bad_ != 1;
    if (guarded) {
        // (a second pass has its own flags: its blocks are tested whatever the first one's hold)
        a.guard = fxGuard(n_, g_flagged_ && !g2_fx_ ? fx_flags_.get() : nullptr);
        if (mode == kSolveFit && g2_fx_) a.guard.lim2 = fx_lim_.get() + p_;
    }
    check(launch_solve(a, &nb, stream_), "solve");
    synchronize();
    if (fx) fxCheck();
    if (guarded && guard_hit_) {
        const RowBlocks marked = guardBlocks(m_);
        contractRows(z_.get(), m_, g_.get(), m_, bw, adaptive, kernel, mode == kSolveCV, 1, marked);
        if (a.guard.lim2) contractRows(z_.get(), mm_, g2_.get(), mm_, bw, adaptive, kernel, false, 2, marked);
        a.guard = FxGuard{};
        check(launch_solve(a, &nb, stream_), "solve");
        stats_.kernel_launches += 1;
        synchronize();
    }
    for (int q = 0; q < 4; q++) out[q] = host_sums_[q];
    {
        int serr = 0;
        std::memcpy(&serr, host_sums_ + 5, sizeof(int));
        if (serr) throw CudaError("adaptive threshold select failed (code " + std::to_string(serr) + ")");
    }
    if (mixed) {
        int err = 0;
        std::memcpy(&err, host_sums_ + 4, sizeof(int));
        if (err) {
            // clear the flag so that the engine's next call starts clean
            check(cudaMemsetAsync(err_.get(), 0, sizeof(int), stream_), "memset err");
            synchronize();
            throw CudaError("tensor-core contraction: a bounded wait timed out");
        }
        out[1] *= s_y_ * s_y_;  // RSS / CV in the units of y
    }
}

// One refinement step of every local solve (mixed path): residual of the
// normal equations over the contraction's FP32 weights (exact sums, or the double-float
// pass where those do not apply), then beta += A~^-1 r.
void Engine::refine(double bw, bool adaptive, int kernel, double out[4])
{
    RefineArgs r{};
    r.n = n_;
    r.p = p_;
    r.ntiles = ntiles32_;
    r.kernel = kernel;
    r.skip = 1;
    r.pts = pts32_.get();
    r.tb = tbsel_.get();
    r.X = xs_.get();
    r.y = ys_.get();
    r.beta = beta_.get();
    r.thr = adaptive ? thr32_.get() : nullptr;
    r.bw = (float)bw;
    r.r = rvec_.get();
    // geographic: the contraction's distances from the device's distance cache, as the contraction read them
    DeviceD2Cache& dc = device_d2c(device_);
    std::unique_lock<std::mutex> d2lock(dc.mu, std::defer_lock);
    if (geographic_ && d2c_limit_bytes_ != 0) {
        d2lock.lock();
        r.d2c = ensureDistanceCache();
        if (!r.d2c) d2lock.unlock();
    }
    // the residuals that the fixed-point sums give, but of rows where a column rests on
    // weights near 2^-62 (FxLimits), which the double-float pass holds in full
    if (refineFx((float)bw, adaptive, kernel, r.d2c)) r.low = refine_low_.get();
    check(launch_refine_residual(r, geographic_, stream_), "refine residual");
    stats_.kernel_launches += 1;
    if (r.d2c) {
        check(cudaEventRecord(dc.used, stream_), "cudaEventRecord");
        d2lock.unlock();
    }
    solve(kSolveRefine, bw, adaptive, kernel, out);
}

double Engine::criterion(double bw, bool adaptive, int kernel, int crit)
{
    if (n_ == 0) throw std::logic_error("no data");
    check(cudaSetDevice(device_), "cudaSetDevice");
    if (precision_ == kMixed) ensureMixed();
    computeThresholds(bw, adaptive);
    if (precision_ == kMixed)
        contractMixed(g_.get(), m_, m_, bw, adaptive, kernel, crit == kCV, 1);
    else
        contract(z_.get(), m_, g_.get(), m_, bw, adaptive, kernel, crit == kCV, 1);
    double s[4];
    solve(crit == kCV ? kSolveCV : kSolveAIC, bw, adaptive, kernel, s);
    if (precision_ == kMixed && refine_search_ && crit == kAIC && s[3] == 0.0) {
        // refine beta (and so RSS); the CV criterion excludes w_ii and is not refined
        double r[4];
        for (int it = 0; it < refine_steps_; it++) refine(bw, adaptive, kernel, r);
        if (refine_steps_ > 0) s[1] = r[1];
    }
    stats_.criterion_evals++;
    if (s[3] > 0.0) return DBL_MAX;
    if (crit == kCV) return std::isfinite(s[1]) ? s[1] : DBL_MAX;
    double v = aicc((double)n_, s[1], s[0]);
    return std::isfinite(v) ? v : DBL_MAX;
}

void Engine::fit(double bw, bool adaptive, int kernel, bool storeS, FitOutput& out)
{
    if (n_ == 0) throw std::logic_error("no data");
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int n = n_, p = p_;
    g2_.alloc((size_t)n * mm_);
    vvec_.alloc((size_t)n * p);
    bse_.alloc((size_t)n * p);
    qdiag_.alloc(n);
    const bool mixed = precision_ == kMixed;
    if (mixed) ensureMixed();
    computeThresholds(bw, adaptive);
    if (mixed) {
        contractMixed(g_.get(), m_, m_, bw, adaptive, kernel, false, 1);
        contractMixed(g2_.get(), mm_, mm_, bw, adaptive, kernel, false, 2);
    } else {
        WeightScope scope{*this};
        contract(z_.get(), m_, g_.get(), m_, bw, adaptive, kernel, false, 1, WeightUse::kKept);
        contract(z_.get(), mm_, g2_.get(), mm_, bw, adaptive, kernel, false, 2, WeightUse::kAgain);
    }
    double s[4];
    solve(kSolveFit, bw, adaptive, kernel, s);
    if (s[3] > 0.0) throw NotSPDError("inv_sympd(): matrix is singular or not positive definite");
    if (mixed) {
        double r[4];
        for (int it = 0; it < refine_steps_; it++) refine(bw, adaptive, kernel, r);
        if (refine_steps_ > 0) s[1] = r[1];
    }
    // S: n x n when stored (isStoreS, GWRBasic.h:708), else only the last
    // location's row, which is what S.row(0) holds after the reference's loop
    int last_sorted = 0;
    for (int sidx = 0; sidx < n; sidx++)
        if (perm_[sidx] == n - 1) last_sorted = sidx;
    S_.alloc(storeS ? (size_t)n * n : (size_t)n);
    check(cudaMemsetAsync(S_.get(), 0, sizeof(double) * S_.size(), stream_), "memset S");
    check(launch_tile_far_thr(n, kTile, geographic_, thrPtr(adaptive), bw, tile_thr16_.get(), stream_), "tile thr");
    stats_.kernel_launches += 2;  // tile thresholds and the hat pass
    if (mixed) {
        if (adaptive) check(launch_to_float(n_, thr_.get(), thr32_.get(), stream_), "thr32");
        HatMixedArgs a{};
        a.n = n;
        a.pts = pts32_.get();
        a.tb16 = tb16_.get();
        a.tile_thr = tile_thr16_.get();
        a.X = xs_.get();
        a.p = p;
        a.v = vvec_.get();
        a.thr32 = adaptive ? thr32_.get() : nullptr;
        a.bw = (float)bw;
        a.kernel = kernel;
        a.S = storeS ? S_.get() : nullptr;
        a.perm = d_perm_.get();
        a.row_target = storeS ? -1 : last_sorted;
        a.s_row = storeS ? nullptr : S_.get();
        const int nsplit = hat_splits(n, num_sms_);
        hat_sum_.alloc((size_t)n * nsplit);
        a.qsum = hat_sum_.get();
        // geographic: the contraction's distances from the device's distance cache, as the contraction read them
        DeviceD2Cache& dc = device_d2c(device_);
        std::unique_lock<std::mutex> d2lock(dc.mu, std::defer_lock);
        if (geographic_ && d2c_limit_bytes_ != 0) {
            d2lock.lock();
            a.d2c = ensureDistanceCache();
            if (!a.d2c) d2lock.unlock();
        }
        check(launch_hat_mixed(a, geographic_, nsplit, qdiag_.get(), stream_), "hat pass");
        if (a.d2c) {
            check(cudaEventRecord(dc.used, stream_), "cudaEventRecord");
            d2lock.unlock();
        }
        stats_.kernel_launches += nsplit > 1 ? 1 : 0;
    } else {
        hatPass(bw, adaptive, kernel, storeS ? S_.get() : nullptr, storeS ? -1 : last_sorted, storeS ? nullptr : S_.get());
    }
    // every result in the original order on the device, then straight into the caller's arrays
    const size_t np = (size_t)n * p;
    out_.alloc(2 * np + n);
    UnpermuteArgs u{};
    u.n = n;
    u.perm = d_perm_.get();
    u.p[0] = u.p[1] = p;
    u.p[2] = 1;
    u.src[0] = beta_.get();
    u.src[1] = bse_.get();
    u.src[2] = qdiag_.get();
    u.dst[0] = out_.get();
    u.dst[1] = out_.get() + np;
    u.dst[2] = out_.get() + 2 * np;
    u.musc = mixed ? musc_.get() : nullptr;
    u.s_y = s_y_;
    u.mu_y = mu_y_;
    u.icol = intercept_col_;
    check(launch_unpermute(u, 3, stream_), "unpermute");
    stats_.kernel_launches += 1;
    out.betas.resize(np);
    out.betasSE.resize(np);
    out.qdiag.resize(n);
    out.S.resize(S_.size());
    out.sRows = storeS ? n : 1;
    auto fetch = [&](double* dst, const double* src, size_t count) {
        check(cudaMemcpyAsync(dst, src, sizeof(double) * count, cudaMemcpyDeviceToHost, stream_), "D2H");
    };
    fetch(out.betas.data(), out_.get(), np);
    fetch(out.betasSE.data(), out_.get() + np, np);
    fetch(out.qdiag.data(), out_.get() + 2 * np, n);
    fetch(out.S.data(), S_.get(), S_.size());
    synchronize();
    out.shat[0] = s[0];
    out.shat[1] = s[2];
    out.rss = s[1];
}

double Engine::golden(bool adaptive, int kernel, int crit, double lower, double upper,
                      std::map<double, double>& record)
{
    double xopt = 0.0;
    golden_section(
        lower, upper, adaptive, [&](double b) { return criterion(b, adaptive, kernel, crit); }, [] { return true; },
        xopt, record);
    return xopt;
}

size_t Engine::estimateBytes(int n, int p, bool geographic, bool mixed, bool adaptive, long long hist_limit,
                             int num_sms)
{
    const double N = n, P = p;
    const double m = P * (P + 1) / 2 + P, mm = P * (P + 1) / 2;
    const double npad = std::ceil(m / 16) * 16;
    const double t16 = std::ceil(N / 16), t32 = std::ceil(N / 32);
    const double g = geographic ? 1.0 : 0.0;
    double b = 8 * N * (2 + 5 * g);                                  // u, v, uR, vR, unit vectors
    b += 8 * N * (P + 1 + 2 * m + 3 + P + 2 + P);                    // x, y, z, g, thr, sel0/1, beta, sii, resid, rvec
    b += 8 * 16384 + 64;                                              // partials, sums
    b += 32 * t16 * (1 + g) + 32 * t32 * (1 + g);                     // tile boxes and caps (16 and 32 points)
    b += 16 * t32 * 32 * (1 + g) + 16 * t32 + 20 * t16;               // point records, tile bounds, tile thresholds
    b += 8 * 256 * m + 8 * 4 * kMaxP * 65;                            // variable-selection scratch
    const double n128 = std::ceil(N / 128) * 128;                    // rows of the contraction's sums
    b += 8 * N * (P + 3) + 28 * N;                                    // the caller's arrays, the ordering's scratch
    if (mixed) {
        b += 8 * N * (P + 1 + m) + t32 * 2 * npad * 128 + 4 * N + 12 * std::ceil(N / 256) * (P + 1);
        // sums and their splits at any number of visited tiles, 64 tiles a chunk
        int splits = 1;
        for (int visits = 64; visits < (int)t32 + 64; visits += 64)
            splits = std::max(splits, tc_splits((int)(n128 / 128), std::min(visits, (int)t32), 64, num_sms));
        b += 12 * n128 * npad * splits;
    }
    b += 8 * N * (mm + 2 * P + 2) + 8 * N * (2 * P + 1) + 4 * N;      // fit: G2, v, betasSE, qDiag, S row, results
    b += 4 * N;                                                       // deferred rows of the exact select
    {
        // FP64 hat pass and fixed-point contraction: rows, split sums, digit images of Z,
        // coordinates (a mixed engine holds them too once it predicts)
        int groups = 0;
        const int w = fx_columns((int)m, &groups);
        int splits = 1;  // of a first pass (one group's rows) and of passes that read kept weights
        for (int g = 1; g <= groups; g++)
            splits = std::max(splits, fx_splits((n + 127) / 128 * g, (n + 15) / 16, num_sms));
        b += 40 * N + 8 * N * hat_splits(n, num_sms);
        b += t16 * groups * w * 256 + std::ceil(N / 1024) * groups * w * 20 + 32 * N;
        // their splits' sums, or those of the blocks that FP64 sums replace (contract64_splits)
        const double blocks = std::ceil(N / kRowBlock), ctas = std::min(16 * blocks, 4.0 * num_sms + std::min(blocks, 4.0 * num_sms));
        const double marked = 8.0 * kRowBlock * std::min(256.0, m) * ctas;
        b += std::max(splits > 1 ? 8 * N * m * splits : 0.0, marked) + 4 * N * splits + N;
    }
    if (adaptive) {
        const double h = 4.0 * (4096 + 64) * N;  // histograms and their segment counts
        if (hist_limit < 0 || h <= (double)hist_limit) b += h;
        b += 64 * 8 * N;                                              // cached order statistics
    }
    return (size_t)(b * 1.05) + (16u << 20);
}

void Engine::predict(int nr, const double* locations, double bw, bool adaptive, int kernel,
                     std::vector<double>& betas)
{
    if (n_ == 0) throw std::logic_error("no data");
    if (nr < 1) throw std::invalid_argument("no prediction locations");
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int p = p_;
    // prediction points in Hilbert order (for compact focus blocks)
    double umin = locations[0], umax = umin, vmin = locations[nr], vmax = vmin;
    for (int i = 0; i < nr; i++) {
        umin = std::min(umin, locations[i]);
        umax = std::max(umax, locations[i]);
        vmin = std::min(vmin, locations[nr + i]);
        vmax = std::max(vmax, locations[nr + i]);
    }
    const double su = umax > umin ? 2147483647.0 / (umax - umin) : 0.0;
    const double sv = vmax > vmin ? 2147483647.0 / (vmax - vmin) : 0.0;
    pf_raw_.alloc(2 * (size_t)nr);
    pf_perm_.alloc(nr);
    std::vector<int> perm;
    check(cudaMemcpyAsync(pf_raw_.get(), locations, sizeof(double) * 2 * nr, cudaMemcpyHostToDevice, stream_), "H2D");
    orderPoints(nr, locations, pf_raw_.get(), umin, su, vmin, sv, pf_perm_.get(), perm);
    pf_u_.alloc(nr);
    pf_v_.alloc(nr);
    pf_uR_.alloc(nr);
    pf_vR_.alloc(nr);
    check(launch_gather_points(nr, pf_raw_.get(), pf_perm_.get(), geographic_, pf_u_.get(), pf_v_.get(), pf_uR_.get(),
                               pf_vR_.get(), stream_),
          "gather points");
    stats_.kernel_launches += 1;
    // the focus bounds share the data's planar frame; widen the slack to cover both
    double slack = slack_;
    if (!geographic_) {
        double maxabs = 0.0;
        for (int s = 0; s < nr; s++)
            maxabs = std::max(maxabs, std::max(std::fabs(locations[s] - uc_), std::fabs(locations[nr + s] - vc_)));
        slack = std::max(slack, std::ldexp(maxabs, -20));
    }
    const int ft16 = (nr + kTile - 1) / kTile, ft32 = (nr + 31) / 32;
    pf_pts_.alloc((size_t)ft32 * 32 * (geographic_ ? 2 : 1));
    pf_tb16_.alloc(ft16);
    std::vector<double> fe;
    if (!geographic_) {
        check(launch_planar_proxy(nr, pf_u_.get(), pf_v_.get(), uc_, vc_, slack, nullptr, nullptr, pf_tb16_.get(), nullptr,
                                  nullptr, pf_pts_.get(), stream_),
              "planar records and bounds");
        stats_.kernel_launches += 1;
    } else {
        std::vector<double> fuR(nr), fvR(nr);
        auto down = [&](std::vector<double>& dst, const double* src) {
            check(cudaMemcpyAsync(dst.data(), src, sizeof(double) * nr, cudaMemcpyDeviceToHost, stream_), "D2H");
        };
        down(fuR, pf_uR_.get());
        down(fvR, pf_vR_.get());
        synchronize();
        fe = unit_vectors(fuR, fvR);
        const std::vector<float4> fpts = point_records(fe);
        const std::vector<float4> ftb = tile_bounds(fe, kTile);
        pf_e_.alloc(fe.size());
        check(cudaMemcpyAsync(pf_e_.get(), fe.data(), sizeof(double) * fe.size(), cudaMemcpyHostToDevice, stream_),
              "H2D unit vectors");
        check(cudaMemcpyAsync(pf_pts_.get(), fpts.data(), sizeof(float4) * fpts.size(), cudaMemcpyHostToDevice, stream_),
              "H2D");
        check(cudaMemcpyAsync(pf_tb16_.get(), ftb.data(), sizeof(float4) * ftb.size(), cudaMemcpyHostToDevice, stream_),
              "H2D");
        synchronize();
    }
    DevPoints F;
    F.n = nr;
    F.u = pf_u_.get();
    F.v = pf_v_.get();
    F.uR = geographic_ ? pf_uR_.get() : nullptr;
    F.vR = geographic_ ? pf_vR_.get() : nullptr;
    F.e = geographic_ ? pf_e_.get() : nullptr;

    // thresholds: fixbw of BandwidthWeight.cpp:40-53 over each location's distances to the data
    const double* thr = nullptr;
    if (adaptive) {
        pf_thr_.alloc(nr);
        pf_d0_.alloc(nr);
        auto select = [&](unsigned rank, double* out) {
            SelectArgs a{};
            a.n = n_;
            a.ntiles = ntiles32_;
            a.P = points();
            a.pts = pts32_.get();
            a.tb = tbsel_.get();
            a.stb = stb_.get();
            a.hist_cache = nullptr;
            a.cache_valid = 0;
            a.rank = rank;
            a.dlo = dlo_;
            a.dhi = dhi_;
            a.eps = sel_eps_;
            a.delta = sel_delta_;
            a.out = out;
            a.err = sel_err_.get();
            a.F = F;
            a.fpts = pf_pts_.get();
            if (geographic_) {
                pf_defer_.alloc(nr);
                a.defer = pf_defer_.get();
                stats_.kernel_launches += 1;
            }
            check(launch_select(a, geographic_, true, num_sms_, stream_), "predict select");
            stats_.kernel_launches += 1;
        };
        const double dn = bw / n_;
        if (dn < 1) {
            const double b0 = std::floor(bw), bx = bw - b0;
            const long long r0 = (long long)(int)b0;
            if (r0 < 1 || r0 >= n_) throw std::out_of_range("Mat::operator(): index out of bounds");
            select((unsigned)r0, pf_d0_.get());
            const double* d1 = nullptr;
            if (bx != 0.0) {
                pf_d1_.alloc(nr);
                select((unsigned)(r0 + 1), pf_d1_.get());
                d1 = pf_d1_.get();
            }
            check(launch_threshold_combine_rows(nr, n_, bw, pf_d0_.get(), d1, pf_thr_.get(), stream_), "threshold");
        } else {
            select((unsigned)n_, pf_d0_.get());
            check(launch_threshold_combine_rows(nr, n_, bw, pf_d0_.get(), nullptr, pf_thr_.get(), stream_),
                  "threshold");
        }
        stats_.kernel_launches += 1;
        thr = pf_thr_.get();
    }
    // X^T W_i X, X^T W_i y at every location, then beta_i = (X^T W_i X)^-1 X^T W_i y
    pf_g_.alloc((size_t)nr * m_);
    bool fx = fxReady(bw, adaptive, kernel), fexact = ixy_exact_;
    FxLimits limits{};
    if (fx) limits = fxLimits(bw, adaptive, kernel, 1);
    if (fx && geographic_ && withinCap(fe)) {
        pf_ie3_.alloc(nr);
        check(launch_int_vectors(nr, pf_uR_.get(), pf_vR_.get(), pf_ie3_.get(), stream_), "integer unit vectors");
        contractFx(pf_ie3_.get(), pf_tb16_.get(), nr, m_, pf_g_.get(), m_, thr, bw, kernel, false, 1, true, limits);
    } else if (fx && !geographic_ && integerCoords(nr, pf_u_.get(), pf_v_.get(), pf_ixy_, fexact)) {
        contractFx(pf_ixy_.get(), pf_tb16_.get(), nr, m_, pf_g_.get(), m_, thr, bw, kernel, false, 1, fexact,
                   limits);
    } else {
        fx = false;
    }
    const auto contractFocus = [&](const RowBlocks& blocks) {
        for (int c0 = 0; c0 < m_; c0 += 256) {  // at most 256 columns a launch
            check(launch_contract64_focus(points(), tb16_.get(), F, pf_tb16_.get(), geographic_, z_.get() + c0, m_,
                                          std::min(256, m_ - c0), pf_g_.get() + c0, m_, thr, bw, kernel, false, 1, true,
                                          stream_, blocks),
                  "predict contraction");
            stats_.kernel_launches += 1;
        }
    };
    contractFocus(fx ? RowBlocks{fx_flags_.get(), fx_state_.get(), nullptr, 0, 0, nullptr} : RowBlocks{});
    pf_beta_.alloc((size_t)nr * p);
    SolveArgs a{};
    a.n = nr;
    a.p = p;
    a.mode = kSolvePredict;
    a.kernel = kernel;
    a.G = pf_g_.get();
    a.ldg = m_;
    a.thr = thr;
    a.bw = bw;
    a.beta = pf_beta_.get();
    a.partials = partials_.get();
    a.tcol = -1;
    int nb = 0;
    a.out = criterionOut();
    if (!fx) a.out.fx_state = nullptr;
    if (fx) a.guard = fxGuard(nr, fx_flags_.get());
    UnpermuteArgs un{};
    un.n = nr;
    un.perm = pf_perm_.get();
    un.p[0] = p;
    un.src[0] = pf_beta_.get();
    out_.alloc((size_t)nr * p);
    un.dst[0] = out_.get();
    betas.resize((size_t)nr * p);
    const auto solveAll = [&] {
        check(launch_solve(a, &nb, stream_), "predict solve");
        check(launch_unpermute(un, 1, stream_), "unpermute");
        stats_.kernel_launches += 4;
        check(cudaMemcpyAsync(betas.data(), out_.get(), sizeof(double) * betas.size(), cudaMemcpyDeviceToHost, stream_),
              "D2H");
        synchronize();
    };
    solveAll();
    if (fx) {
        fxCheck();
        if (guard_hit_) {
            contractFocus(guardBlocks(m_));
            a.guard = FxGuard{};
            solveAll();
        }
    }
    int serr = 0;
    std::memcpy(&serr, host_sums_ + 5, sizeof(int));
    if (serr) throw CudaError("adaptive threshold select failed (code " + std::to_string(serr) + ")");
    if (host_sums_[3] > 0.0) throw NotSPDError("inv_sympd(): matrix is singular or not positive definite");
}

void Engine::releaseDistanceCache()
{
    DeviceD2Cache& c = device_d2c(device_);
    std::lock_guard<std::mutex> lk(c.mu);
    d2c_valid_ = false;
    if (c.owner != this) return;
    check(cudaSetDevice(device_), "cudaSetDevice");
    free_d2c(c);
}

bool Engine::distanceCacheActive() const
{
    DeviceD2Cache& c = device_d2c(device_);
    std::lock_guard<std::mutex> lk(c.mu);
    return c.owner == this && d2c_valid_;
}

// The device's distance cache holding this dataset, filled now if needed, or
// null when the cache does not apply or does not fit.  The caller holds the
// cache's lock and records its `used` event after the launch that reads it.
const float* Engine::ensureDistanceCache()
{
    DeviceD2Cache& c = g_d2c[device_];
    if (c.owner == this && d2c_valid_ && c.ptr) return c.ptr;
    float* d2c = acquireDistanceCache();
    if (!d2c) return nullptr;
    cudaEvent_t e0 = stats_on_ ? timerBegin() : nullptr;
    fill_scratch_.alloc((size_t)(n_ + 127) / 128 + 2);
    check(launch_fill_d2_sym(n_, pts32_.get(), d2c, fill_scratch_.get(), num_sms_, stream_), "fill distance cache");
    stats_.kernel_launches += 2;
    if (stats_on_) {
        timerEnd(e0, 2);
        stats_.d2c_fills += 1;
    }
    d2c_valid_ = true;
    return d2c;
}

// The device's distance cache, owned by this engine and large enough for its
// dataset (contents not yet this dataset's: the caller fills it), or null.
// The caller holds the cache's lock.
float* Engine::acquireDistanceCache()
{
    if (!geographic_ || precision_ != kMixed || d2c_limit_bytes_ == 0 || n_ < 1) return nullptr;
    DeviceD2Cache& c = g_d2c[device_];
    d2c_valid_ = false;
    const size_t need = d2_cache_bytes(n_);
    if (d2c_limit_bytes_ > 0 && need > (size_t)d2c_limit_bytes_) return nullptr;
    if (c.bytes < need) {
        if (c.ptr) free_d2c(c);
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        const size_t reserve = std::max((size_t)16 << 30, total_b / 8);
        if (need + reserve > free_b && release_idle_scratch()) cudaMemGetInfo(&free_b, &total_b);
        if (need + reserve > free_b) return nullptr;
        if (cudaMalloc(&c.ptr, need) != cudaSuccess) {
            cudaGetLastError();  // too little memory after all: run without the cache
            c.ptr = nullptr;
            return nullptr;
        }
        c.bytes = need;
        c.owner = nullptr;
    }
    if (!c.used) check(cudaEventCreateWithFlags(&c.used, cudaEventDisableTiming), "cudaEventCreate");
    // the previous owner's launches that read the buffer come first
    if (c.owner && c.owner != this) check(cudaStreamWaitEvent(stream_, c.used, 0), "cudaStreamWaitEvent");
    c.owner = this;
    return c.ptr;
}

void Engine::clearCaches()
{
    d2c_valid_ = false;
    recycleRanks();
    hist_valid_ = false;
    thr_valid_ = false;
    gall_valid_ = false;
}

void Engine::recordEvent(int slot)
{
    if (slot < 0 || slot >= 8) throw std::invalid_argument("event slot out of range");
    check(cudaSetDevice(device_), "cudaSetDevice");
    if (!events_[slot]) check(cudaEventCreate(&events_[slot]), "cudaEventCreate");
    check(cudaEventRecord(events_[slot], stream_), "cudaEventRecord");
}

float Engine::elapsedMs(int a, int b)
{
    if (a < 0 || a >= 8 || b < 0 || b >= 8 || !events_[a] || !events_[b])
        throw std::invalid_argument("event slot not recorded");
    check(cudaEventSynchronize(events_[b]), "cudaEventSynchronize");
    float ms = 0.f;
    check(cudaEventElapsedTime(&ms, events_[a], events_[b]), "cudaEventElapsedTime");
    return ms;
}

double Engine::globalCriterion(const std::vector<int>& cols) { return globalCriteria({cols})[0]; }

std::vector<double> Engine::globalCriteria(const std::vector<std::vector<int>>& subsets)
{
    if (n_ == 0) throw std::logic_error("no data");
    const int count = (int)subsets.size();
    if (count < 1 || count > kMaxP) throw std::invalid_argument("number of column subsets out of range");
    SubsetList list{};
    list.count = (int)subsets[0].size();
    if (list.count < 1 || list.count > kMaxP) throw std::invalid_argument("column subset size out of range");
    for (int s = 0; s < count; s++) {
        if ((int)subsets[s].size() != list.count) throw std::invalid_argument("column subsets differ in size");
        for (int a = 0; a < list.count; a++) {
            if (subsets[s][a] < 0 || subsets[s][a] >= p_) throw std::invalid_argument("column index out of range");
            list.cols[s][a] = (unsigned char)subsets[s][a];
        }
    }
    check(cudaSetDevice(device_), "cudaSetDevice");
    const int blocks = global_criteria_blocks(n_);
    if (!gall_valid_) {
        const int nb = 256;
        gall_.alloc(m_);
        gall_part_.alloc(std::max((size_t)nb * m_, (size_t)kMaxP * 64 * 4));
        check(launch_column_sums(n_, m_, z_.get(), gall_part_.get(), nb, gall_.get(), stream_), "column sums");
        std::vector<int> first(kMaxP + 1);
        for (int s = 0; s <= kMaxP; s++) first[s] = s * blocks;
        gfirst_.alloc(first.size());
        check(cudaMemcpyAsync(gfirst_.get(), first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice, stream_),
              "H2D");
        gsub_.alloc(4 * kMaxP);
        synchronize();
        gall_valid_ = true;
    }
    check(launch_global_criteria(n_, p_, list, count, x_.get(), y_.get(), gall_.get(), gall_part_.get(), gfirst_.get(),
                                 gsub_.get(), stream_),
          "global criteria");
    stats_.kernel_launches += 2;
    std::vector<double> sums(4 * count), out(count);
    check(cudaMemcpyAsync(sums.data(), gsub_.get(), sizeof(double) * sums.size(), cudaMemcpyDeviceToHost, stream_),
          "D2H sums");
    synchronize();
    for (int s = 0; s < count; s++) {
        const double v = aicc((double)n_, sums[4 * s + 1], sums[4 * s]);
        out[s] = sums[4 * s + 3] > 0.0 || !std::isfinite(v) ? DBL_MAX : v;
    }
    return out;
}

double Engine::maxDistance()
{
    check(cudaSetDevice(device_), "cudaSetDevice");
    check(cudaMemsetAsync(key_.get(), 0, 2 * sizeof(unsigned long long), stream_), "memset");
    if (geographic_) rowmax_.alloc(n_);
    check(launch_max_distance(points(), geographic_, boxes32_.get(), caps32_.get(), key_.get(), rowmax_.get(), num_sms_,
                              stream_), "maxdist");
    unsigned long long k = 0;
    check(cudaMemcpyAsync(&k, key_.get() + (geographic_ ? 1 : 0), sizeof(k), cudaMemcpyDeviceToHost, stream_),
          "D2H");
    synchronize();
    uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}

void Engine::thresholds(double bw, bool adaptive, std::vector<double>& out)
{
    check(cudaSetDevice(device_), "cudaSetDevice");
    out.assign(n_, bw);
    if (!adaptive) return;
    computeThresholds(bw, adaptive);
    std::vector<double> h(n_);
    int serr = 0;
    check(cudaMemcpyAsync(h.data(), thr_.get(), sizeof(double) * n_, cudaMemcpyDeviceToHost, stream_), "D2H");
    check(cudaMemcpyAsync(&serr, sel_err_.get(), sizeof(int), cudaMemcpyDeviceToHost, stream_), "D2H");
    synchronize();
    if (serr) throw CudaError("adaptive threshold select failed (code " + std::to_string(serr) + ")");
    for (int s = 0; s < n_; s++) out[perm_[s]] = h[s];
}

}  // namespace gwgpu
