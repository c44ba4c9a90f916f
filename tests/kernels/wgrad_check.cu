// The weight-gradient kernels by themselves, launched as the network launches
// them, against sums over the voxels on the host.
//   wgrad_check exact : small whole numbers, whose sums are exact in FP32 in
//                       any order; counts the sums that differ.
//   wgrad_check inf   : an infinity in one operand; counts the sums that differ
//                       (all NaN are alike) from IEEE sums over the pairs of
//                       voxels that the convolution has.
//   wgrad_check bias  : random positive gradients; the largest relative error
//                       of a bias gradient against FP64.
#include "sf_unet.cu"

#include <cstdio>
#include <cstring>

using sfb::Dims;
namespace net = sfb::net;

namespace {

uint32_t state = 12345u;
uint32_t rnd() { return state = state * 1664525u + 1013904223u, state >> 8; }

struct Tensor {
    Dims d;
    int channels;
    std::vector<float> h;
    __nv_bfloat16* dev = nullptr;
    Tensor(Dims dims, int c) : d(dims), channels(c), h(static_cast<size_t>(dims.nx) * dims.ny * dims.nz * c) {}
    Tensor(const Tensor&) = delete;
    ~Tensor() { cudaFree(dev); }
    float& at(size_t v, int c) { return h[v * channels + c]; }
    bool upload() {
        std::vector<__nv_bfloat16> b(h.size());
        for (size_t i = 0; i < h.size(); ++i) b[i] = __float2bfloat16(h[i]);
        return cudaMalloc(&dev, b.size() * 2) == cudaSuccess && cudaMemcpy(dev, b.data(), b.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess;
    }
};

struct Sums {
    std::vector<float> dw, db;
};

// The kernels' result for one layer; the error word must stay zero.
bool run(Tensor& in, Tensor& out, Sums& r) {
    const int ci = in.channels, co = out.channels;
    r.dw.assign(27u * ci * co, 0.0f);
    r.db.assign(co, 0.0f);
    float* g = nullptr;
    unsigned* error = nullptr;
    const size_t n = r.dw.size() + r.db.size();
    if (!in.upload() || !out.upload() || cudaMalloc(&g, n * 4) != cudaSuccess || cudaMalloc(&error, 4) != cudaSuccess) return false;
    cudaMemset(g, 0, n * 4);
    cudaMemset(error, 0, 4);
    float* const db = g + r.dw.size();
    cudaError_t e;
    if (co == 16) {
        net::ChainLaunch chain;
        chain.add(in.dev, ci, out.dev, g, db, static_cast<long long>(in.h.size()) / ci);
        e = chain.launch(in.d, nullptr, error);
    } else {
        e = net::wgrad_any(ci, co, in.dev, out.dev, g, db, in.d, nullptr, error);
    }
    unsigned failed = 1;
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(r.dw.data(), g, r.dw.size() * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(r.db.data(), db, r.db.size() * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&failed, error, 4, cudaMemcpyDeviceToHost);
    cudaFree(g);
    cudaFree(error);
    if (e != cudaSuccess) std::printf("error %s\n", cudaGetErrorString(e));
    return e == cudaSuccess && failed == 0;
}

// The same on the host: FP32 sums (exact for whole numbers).
void host(Tensor& in, Tensor& out, Sums& r) {
    const int ci = in.channels, co = out.channels;
    const Dims d = in.d;
    r.dw.assign(27u * ci * co, 0.0f);
    r.db.assign(co, 0.0f);
    for (int z = 0; z < d.nz; ++z)
        for (int y = 0; y < d.ny; ++y)
            for (int x = 0; x < d.nx; ++x) {
                const float* const o = &out.at(x + static_cast<size_t>(d.nx) * (y + static_cast<size_t>(d.ny) * z), 0);
                for (int c = 0; c < co; ++c) r.db[c] += o[c];
                for (int t = 0; t < 27; ++t) {
                    const int sx = x + t % 3 - 1, sy = y + t / 3 % 3 - 1, sz = z + t / 9 - 1;
                    if (sx < 0 || sy < 0 || sz < 0 || sx >= d.nx || sy >= d.ny || sz >= d.nz) continue;
                    const float* const i = &in.at(sx + static_cast<size_t>(d.nx) * (sy + static_cast<size_t>(d.ny) * sz), 0);
                    for (int c = 0; c < co; ++c) {
                        float* const w = &r.dw[(static_cast<size_t>(t) * co + c) * ci];
                        for (int k = 0; k < ci; ++k) w[k] += o[c] * i[k];
                    }
                }
            }
}

bool same(float a, float b) { return a == b || (std::isnan(a) && std::isnan(b)); }
long differ(const Sums& a, const Sums& b) {
    long n = 0;
    for (size_t i = 0; i < a.dw.size(); ++i) n += !same(a.dw[i], b.dw[i]);
    for (size_t i = 0; i < a.db.size(); ++i) n += !same(a.db[i], b.db[i]);
    return n;
}

const int kLayers[][2] = {{16, 16}, {48, 16}, {16, 32}, {32, 32}, {96, 32}, {32, 64}, {64, 64}};

}  // namespace

int main(int argc, char** argv) {
    const char* const mode = argc > 1 ? argv[1] : "exact";
    // a voxel, grids below and beyond a tile of 32 x 8 x 2, several tiles a CTA
    // (the last), several segments of the chain kernel with a part of a chunk
    const Dims grids[] = {{1, 1, 1, 0}, {2, 2, 2, 0}, {4, 4, 4, 0}, {7, 3, 2, 0}, {33, 9, 3, 0}, {20, 6, 10, 0}, {10, 26, 5, 0}, {64, 8, 4, 0}, {8, 28, 24, 0}, {48, 20, 40, 0}};
    if (std::strcmp(mode, "bias") == 0) {
        for (const int co : {16, 32, 64}) {
            Tensor in({64, 32, 64, 0}, co == 16 ? 16 : co), out({64, 32, 64, 0}, co);
            std::vector<double> want(co, 0.0);
            for (size_t i = 0; i < out.h.size(); ++i) {
                out.h[i] = __bfloat162float(__float2bfloat16(std::ldexp(1.0f + static_cast<float>(rnd() & 0xffff) / 65536.0f, -static_cast<int>(rnd() % 12))));
                want[i % co] += out.h[i];
            }
            Sums got;
            if (!run(in, out, got)) return 1;
            double worst = 0.0;
            for (int c = 0; c < co; ++c) worst = std::max(worst, std::fabs(got.db[c] - want[c]) / want[c]);
            std::printf("%d %.3e\n", co, worst);
        }
        return 0;
    }
    const bool inf = std::strcmp(mode, "inf") == 0;
    for (const Dims& d : grids) {
        if (inf && (d.nx < 3 || d.ny < 3 || d.nz < 3)) continue;  // no voxel without a neighbour beyond a face
        const size_t voxels = static_cast<size_t>(d.nx) * d.ny * d.nz;
        for (const auto& l : kLayers) {
            if (voxels > 20000 && l[1] != 32) continue;
            for (int form = 0; form < (inf ? 2 : 1); ++form) {
                Tensor in(d, l[0]), out(d, l[1]);
                for (float& v : in.h) v = inf ? static_cast<float>(1 + rnd() % 3) : static_cast<float>(static_cast<int>(rnd() % 7) - 3);
                for (float& v : out.h) v = inf ? static_cast<float>(1 + rnd() % 3) : static_cast<float>(static_cast<int>(rnd() % 7) - 3);
                if (inf && form == 0)  // the last column of `in`, one channel
                    for (size_t v = d.nx - 1; v < voxels; v += d.nx) in.at(v, 5) = INFINITY;
                if (inf && form == 1) {  // a voxel of dout that has all 26 neighbours, just behind the first of the chain's segments where the grid has several
                    size_t at = 1152 + 3;
                    if (voxels != 8 * 28 * 24) at = 1 + static_cast<size_t>(d.nx) * (1 + static_cast<size_t>(d.ny));
                    out.at(at, 2) = INFINITY;
                }
                Sums got, want;
                if (!run(in, out, got)) return 1;
                host(in, out, want);
                std::printf("%dx%dx%d %d->%d form %d: %zu sums, %ld differ\n", d.nx, d.ny, d.nz, l[0], l[1], form, want.dw.size() + want.db.size(), differ(got, want));
            }
        }
    }
    return 0;
}
