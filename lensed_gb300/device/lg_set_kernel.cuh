// set_params module: compiled separately, without FMA contraction and with
// the double-evaluated elementary functions (or the single-precision
// functions that return the same values), so the object data of every
// candidate are the IEEE single-precision values of the plugin formulas.

// ------------------------------------------------------------ set_params --
// Physical parameters (pmap order, double) -> object data (src/nested.c:67-77
// and the generated set_params of src/kernel.c:114-150).  A block takes up to
// LG_SET_PER candidates, one a lane, and gives each object a warp of its own:
// the time is that of the slowest object (a Sersic source) whatever the model
// and, up to 32 candidates, the batch; what bounds it is the latency of that
// one chain.  Objects whose positions carry image-plane priors follow in a
// second phase, once the lenses they are deflected through are set.
// (Before, with FP64 functions: one thread a candidate through all objects, 22.9
// us for 1024 candidates of four objects, now 14.7; a block of a warp an object
// for each candidate of a small batch, 8.4 us for 7, now 6.3.)
#define LG_SET_FIT (40000 / (sizeof(lg_model) + 4 * (LG_NPARS + 1)))
#define LG_SET_PER (LG_SET_FIT < 1 ? 1 : (LG_SET_FIT < 32 ? (int)LG_SET_FIT : 32))
#define LG_SET_WARPS (LG_NOBJ < 16 ? LG_NOBJ : 16)
static_assert(sizeof(lg_model) % 4 == 0, "object data are 32-bit words");

extern "C" __global__ void __launch_bounds__(32 * LG_SET_WARPS)
    lg_set_params_kernel(const double* __restrict__ params, int B, lg_model* __restrict__ models)
{
    __shared__ lg_model m[LG_SET_PER];
    __shared__ float p[LG_SET_PER][LG_NPARS + 1];
    const int b0 = blockIdx.x * LG_SET_PER;
    const int n = B - b0 < LG_SET_PER ? B - b0 : LG_SET_PER;
    const int warp = threadIdx.x / 32, c = threadIdx.x % 32;
    const int words = n * (int)(sizeof(lg_model) / 4);
    // padding included: object data compare byte for byte
    for (int i = threadIdx.x; i < words; i += blockDim.x) reinterpret_cast<unsigned*>(m)[i] = 0;
    if (warp == 0 && c < n) lg_load_params(params + (size_t)(b0 + c) * LG_NPARS, p[c]);
    __syncthreads();
    for (int phase = 0; phase < 2; ++phase) {
        if (c < n)
            for (int w = warp; w < LG_NOBJ; w += LG_SET_WARPS)
                if (lg_obj_phase[w] == phase) lg_set_object(m[c], p[c], w);
        __syncthreads();
    }
    const unsigned* src = reinterpret_cast<const unsigned*>(m);
    unsigned* dst = reinterpret_cast<unsigned*>(models + b0);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

extern "C" __device__ const unsigned lg_model_bytes = sizeof(lg_model);
extern "C" __device__ const int lg_set_shape[2] = {LG_SET_PER, 32 * LG_SET_WARPS};  // candidates, threads a block
