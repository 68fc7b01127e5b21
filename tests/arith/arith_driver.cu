// Applies one of the library's device arithmetic functions to pairs of doubles:
//   arith_driver OP IN OUT    IN: n pairs (x, y); OUT: n pairs
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "gcv_leaf64.cuh"
#include "gcv_setup.cuh"

using namespace gcv;

__global__ void k_apply(int op, const double2* in, double2* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x = in[i].x;
    int s = (int)in[i].y;
    double2 r = make_double2(0.0, 0.0);
    float corr = 0.0f;
    ff f{0.0f, 0.0f};
    switch (op) {
    case 0: r.x = n_recip(x); break;
    case 1:
        r.x = kronrod_root(x, 1.0f, corr);
        r.y = (double)corr;
        break;
    case 4: f = ff_recip(ff_from_double(x)); break;
    case 5: r.x = double_of_fix(fix_of_double(x)); break;
    case 6: r.x = double_of_fix(fix_of_float((float)x)); break;
    case 7: f = ff_from_double_scaled(x, s); break;
    case 8: r.x = scale_exp(x, s); break;
    case 9: r.x = double_of_float((float)x); break;
    case 10:
        lift_denormal(x, s);
        r = make_double2(x, (double)s);
        break;
    case 11: r.x = (double)scale_down((float)x, s); break;
    default: break;
    }
    if (op == 4 || op == 7) r = make_double2((double)f.hi, (double)f.lo);
    out[i] = r;
}

int main(int argc, char** argv)
{
    if (argc != 4) return 2;
    FILE* f = fopen(argv[2], "rb");
    if (!f) return 3;
    fseek(f, 0, SEEK_END);
    const size_t n = (size_t)ftell(f) / sizeof(double2);
    rewind(f);
    std::vector<double2> h(n);
    if (fread(h.data(), sizeof(double2), n, f) != n) return 4;
    fclose(f);
    double2 *in = nullptr, *out = nullptr;
    if (cudaMalloc(&in, n * sizeof(double2)) || cudaMalloc(&out, n * sizeof(double2))) return 5;
    cudaMemcpy(in, h.data(), n * sizeof(double2), cudaMemcpyHostToDevice);
    k_apply<<<(unsigned)((n + 255) / 256), 256>>>(atoi(argv[1]), in, out, (int)n);
    if (cudaMemcpy(h.data(), out, n * sizeof(double2), cudaMemcpyDeviceToHost) != cudaSuccess) return 6;
    f = fopen(argv[3], "wb");
    if (!f || fwrite(h.data(), sizeof(double2), n, f) != n) return 7;
    fclose(f);
    return 0;
}
