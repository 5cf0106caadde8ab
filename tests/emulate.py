"""Runs the kernels of a generated pipeline on the CPU -- a test aid.

The generated translation unit is compiled by g++ with the address and
undefined-behaviour sanitizers: every thread of a CTA is a fiber, CTAs run
one after another, TMA loads copy the box that their tensor map describes.
Global buffers and shared memory have exactly their size, shared memory
starts out as NaN in every CTA, so what it shows is

* reads and writes outside a buffer, misaligned vector accesses and TMA
  coordinates (the run fails with the sanitizer's report);
* values that no loop computes (NaN, or the pattern the outputs are filled
  with);
* wrong values, against any oracle.

It shows no race: threads run one at a time from barrier to barrier (in
rising or falling order).  Tiny images only."""

import os
import re
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "polymage_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"),
                        "include")

DEVICE = r'''
#include <assert.h>
#include <stdlib.h>
#include <ucontext.h>
#undef __shared__
#undef __launch_bounds__
#undef __grid_constant__
#define __shared__ static
#define __launch_bounds__(...)
#define __grid_constant__
#define blockIdx emu_block
#define gridDim emu_grid
#define threadIdx emu_tid
#define blockDim emu_block_dim
static uint3 emu_tid, emu_block, emu_grid, emu_block_dim;
static unsigned char* emu_smem;
static unsigned emu_threads;
struct emu_fiber { ucontext_t c; char* stack; int at; int done; };
static emu_fiber* emu_f;
static ucontext_t emu_main;
static unsigned emu_cur;
static int emu_or, emu_or_last;
static void (*emu_fn)();
#define EMU_STACK (256 << 10)
// at: 0 runnable, 1 at a CTA barrier, 2 at a warp barrier
static void emu_wait(int what) {
  emu_f[emu_cur].at = what;
  swapcontext(&emu_f[emu_cur].c, &emu_main);
}
static void __syncthreads() { emu_wait(1); }
static void __syncwarp() { emu_wait(2); }
static int __syncthreads_or(int p) { emu_or |= p; emu_wait(1); return emu_or_last; }
static void emu_entry() { emu_fn(); emu_f[emu_cur].done = 1; }
static int emu_order() { const char* e = getenv("EMU_ORDER"); return e ? atoi(e) : 0; }
static void emu_cta(unsigned nt) {
  if (nt > emu_threads) {
    emu_f = (emu_fiber*)realloc(emu_f, sizeof(emu_fiber) * nt);
    for (unsigned i = emu_threads; i < nt; ++i) emu_f[i].stack = (char*)malloc(EMU_STACK);
    emu_threads = nt;
  }
  for (unsigned i = 0; i < nt; ++i) {
    getcontext(&emu_f[i].c);
    emu_f[i].c.uc_stack.ss_sp = emu_f[i].stack;
    emu_f[i].c.uc_stack.ss_size = EMU_STACK;
    emu_f[i].c.uc_link = &emu_main;
    emu_f[i].at = emu_f[i].done = 0;
    makecontext(&emu_f[i].c, emu_entry, 0);
  }
  while (true) {
    unsigned live = 0, cta = 0, ran = 0;
    for (unsigned k = 0; k < nt; ++k) {
      const unsigned i = emu_order() ? nt - 1 - k : k;
      if (emu_f[i].done || emu_f[i].at) continue;
      emu_cur = i;
      emu_tid.x = i;
      ++ran;
      swapcontext(&emu_main, &emu_f[i].c);
    }
    for (unsigned i = 0; i < nt; ++i) { live += !emu_f[i].done; cta += !emu_f[i].done && emu_f[i].at == 1; }
    if (!live) break;
    for (unsigned w = 0; w < nt; w += 32) {
      bool all = true, any = false;
      for (unsigned i = w; i < nt && i < w + 32; ++i) {
        any |= emu_f[i].at == 2;
        all &= emu_f[i].at == 2;
      }
      assert(!any || all);
      for (unsigned i = w; any && i < nt && i < w + 32; ++i) emu_f[i].at = 0;
    }
    if (cta) {
      if (cta == nt) {
        emu_or_last = emu_or; emu_or = 0;
        for (unsigned i = 0; i < nt; ++i) emu_f[i].at = 0;
      } else if (!ran) { fprintf(stderr, "barrier not reached by all\n"); abort(); }
    }
  }
}
template <typename L> static const L* emu_arg_of(const L* set) { static const L* a; if (set) a = set; return a; }
template <typename L> struct emu_kernel { static void (*k)(L); static void call() { k(*emu_arg_of<L>(nullptr)); } };
template <typename L> void (*emu_kernel<L>::k)(L);
template <typename L> static void emu_launch(void (*k)(L), unsigned grid, unsigned nt, size_t smem, const L& arg) {
  emu_kernel<L>::k = k;
  emu_arg_of<L>(&arg);
  emu_grid.x = grid;
  emu_block_dim.x = nt;
  for (unsigned b = 0; b < grid; ++b) {
    emu_smem = (unsigned char*)aligned_alloc(128, smem ? (smem + 127) / 128 * 128 : 128);
    memset(emu_smem, 0xff, smem);
    emu_block.x = b;
    emu_fn = &emu_kernel<L>::call;
    emu_cta(nt);
    free(emu_smem);
  }
}
template <typename L> static cudaError_t pm_launch_pdl(void (*k)(L), unsigned grid, unsigned nt, size_t smem, cudaStream_t, const L& arg, bool) {
  emu_launch(k, grid, nt, smem, arg);
  return cudaSuccess;
}
template <typename T> static T __ldg(const T* p) { return *p; }
template <typename T> static T __ldcg(const T* p) { return *p; }
template <typename T, typename U> static T atomicAdd(T* p, U v) { T o = *p; *p += v; return o; }
template <typename T, typename U> static T atomicOr(T* p, U v) { T o = *p; *p |= v; return o; }
template <typename T, typename U> static T atomicMin(T* p, U v) { T o = *p; if (v < o) *p = v; return o; }
template <typename T, typename U> static T atomicMax(T* p, U v) { T o = *p; if (v > o) *p = v; return o; }
static int atomicCAS(int* p, int c, int v) { int o = *p; if (o == c) *p = v; return o; }
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static cudaError_t emu_symbol(void* d, const void* s, size_t n) { memcpy(d, s, n); return cudaSuccess; }
#define cudaMemcpyFromSymbol(d, s, n) emu_symbol(d, &s, n)
#define cudaMemcpyToSymbol(s, d, n) emu_symbol(&s, d, n)
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor(p, ...) (*(p) = 1, cudaSuccess)
#define cudaGetSymbolAddress(p, s) (*(p) = (void*)&s, cudaSuccess)
static const int emu_sms = 1;
#define cudaFuncSetAttribute(...) cudaSuccess
// the fields of a tensor map that a tiled load uses
struct emu_map { char* base; int rank, es; unsigned long long dim[5], stride[5]; unsigned box[5]; };
static_assert(sizeof(emu_map) <= sizeof(CUtensorMap), "tensor map");
static CUresult emu_encode(CUtensorMap* m, CUtensorMapDataType t, cuuint32_t rank, void* base, const cuuint64_t* dim, const cuuint64_t* st, const cuuint32_t* box, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  emu_map e;
  e.base = (char*)base; e.rank = rank;
  e.es = t == CU_TENSOR_MAP_DATA_TYPE_UINT8 ? 1 : t == CU_TENSOR_MAP_DATA_TYPE_UINT16 ? 2 :
         t == CU_TENSOR_MAP_DATA_TYPE_FLOAT64 || t == CU_TENSOR_MAP_DATA_TYPE_INT64 ? 8 : 4;
  for (unsigned i = 0; i < rank; ++i) { e.dim[i] = dim[i]; e.box[i] = box[i]; e.stride[i] = i ? st[i - 1] : e.es; }
  memcpy((void*)m, &e, sizeof(e));
  return CUDA_SUCCESS;
}
static pm_encode_tiled_fn pm_get_encode_fn() { return emu_encode; }
static long long emu_expect, emu_got;
static void pm_mbar_init(uint64_t*, uint32_t) { emu_expect = emu_got = 0; }
static void pm_mbar_inval(uint64_t*) {}
static void pm_fence_barrier_init() {}
static void pm_fence_proxy_async() {}
static void pm_fence_proxy_async_all() {}
static void pm_grid_dep_wait() {}
static void pm_grid_dep_launch() {}
static void pm_cp_async_wait() {}
// a chain kernel runs as one CTA here, so its own barriers order its phases
static bool pm_grid_sync(unsigned*, unsigned, unsigned*) { __syncthreads(); return true; }
static void pm_mbar_arrive_expect_tx(uint64_t*, uint32_t b) { emu_expect += b; }
// (copies are done when they are issued; the bytes announced have to match)
static bool pm_mbar_wait(uint64_t*, uint32_t, unsigned*) { assert(emu_expect == emu_got); return true; }
template <bool CH, typename T> static void pm_copy(T* dst, const T* src, bool ok) { *dst = ok ? *src : (T)0; }
static void emu_tma(void* dst, const CUtensorMap* m, const int* c) {
  emu_map e;
  memcpy(&e, m, sizeof(e));
  if ((c[0] * e.es) % 16 || ((uintptr_t)dst & 127)) { fprintf(stderr, "misaligned TMA load\n"); abort(); }
  long long n = 1;
  for (int i = 0; i < e.rank; ++i) n *= e.box[i];
  for (long long k = 0; k < n; ++k) {
    long long r = k, off = 0;
    bool in = true;
    for (int i = 0; i < e.rank; ++i) {
      const long long x = c[i] + r % e.box[i];
      r /= e.box[i];
      in &= x >= 0 && x < (long long)e.dim[i];
      off += x * (long long)e.stride[i];
    }
    if (in) memcpy((char*)dst + k * e.es, e.base + off, e.es);
    else memset((char*)dst + k * e.es, 0, e.es);
  }
  emu_got += n * e.es;
}
static void pm_tma_load_1d(void* d, const CUtensorMap* m, uint64_t*, int a) { int c[] = {a}; emu_tma(d, m, c); }
static void pm_tma_load_2d(void* d, const CUtensorMap* m, uint64_t*, int a, int b) { int c[] = {a, b}; emu_tma(d, m, c); }
static void pm_tma_load_3d(void* d, const CUtensorMap* m, uint64_t*, int a, int b, int e) { int c[] = {a, b, e}; emu_tma(d, m, c); }
static void pm_tma_load_4d(void* d, const CUtensorMap* m, uint64_t*, int a, int b, int e, int f) { int c[] = {a, b, e, f}; emu_tma(d, m, c); }
static void pm_tma_load_5d(void* d, const CUtensorMap* m, uint64_t*, int a, int b, int e, int f, int g) { int c[] = {a, b, e, f, g}; emu_tma(d, m, c); }
'''

# the runtime calls that an entry point makes, on host memory
HOST = r'''
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = aligned_alloc(256, (n + 255) / 256 * 256); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = 0; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = 0; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeDevice; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = emu_sms; return cudaSuccess; }
}
int main(int argc, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  void* b[EMU_NBUF];
  for (int i = 0; i < EMU_NBUF; ++i) {
    long long n, shift;
    if (fread(&n, 8, 1, f) != 1 || fread(&shift, 8, 1, f) != 1) return 9;
    char* p = (char*)aligned_alloc(256, (n + shift + 255) / 256 * 256) + (256 - (n + shift) % 256) % 256 / 16 * 16;
    b[i] = p + shift;
    if (n && fread(b[i], 1, n, f) != (size_t)n) return 9;
  }
  fclose(f);
  const int st = EMU_CALL;
  f = fopen(argv[2], "wb");
  EMU_WRITE
  fclose(f);
  return st ? 40 + st : pm_err_word ? 50 : 0;
}
'''


class EmulationError(AssertionError):
    pass


def _device_source(source):
    rt = open(os.path.join(CSRC, "pm_runtime.cuh")).read()
    # functions of inline PTX (and the launch wrapper) are replaced by the
    # emulation's; everything else of the runtime header is kept
    parts = re.split(r"(?m)^(?=(?:template <|static |__device__|__host__|"
                     r"struct |typedef |// ))", rt)
    keep = []
    for p in parts:
        if "asm volatile" in p or "pm_grid_sync" in p or \
                "cudaLaunchKernelEx" in p or "cudaGetDriverEntryPoint" in p \
                or "__cvta_generic_to_shared" in p or \
                re.match(r"__device__ __forceinline__ bool pm_mbar_wait", p):
            continue
        keep.append(p)
    # a template header whose function went away goes too
    text = re.sub(r"(?m)^template <[^\n]*>\n(?=(?:static|__device__|//|"
                  r"template|struct|typedef|\s*$))(?=(?://|template|struct|"
                  r"typedef|\s*$))", "", "".join(keep))
    text = re.sub(r"template <bool CH, typename T>\n$", "", text)
    head, body = text.split("// device helpers", 1)
    head += "// device helpers"
    encode = body.index("typedef CUresult (*pm_encode_tiled_fn)")
    fn_end = body.index(");", encode) + 2
    typedef = body[encode:fn_end]
    body = body[:encode] + body[fn_end:]
    first = head.rindex("// -----")
    source = re.sub(r"extern __shared__ __align__\(128\) unsigned char "
                    r"pm_smem\[\];", "unsigned char* const pm_smem = "
                    "emu_smem;", source)
    source = re.sub(r"([\w]+)<<<([^\n]*?), (\d+), (\d+), s>>>\((\w+)\)",
                    r"emu_launch(\1, \2, \3, \4, \5)", source)
    source = re.sub(r"(\w+_init)<<<([^\n]*?), 256, 0, s>>>\((\w+)\)",
                    r"emu_launch(\1, \2, 256, 0, \3)", source)
    return source.replace('#include "pm_runtime.cuh"',
                          head[:first] + typedef + "\n" + DEVICE +
                          head[first:] + body)


def run(pipeline, params, inputs, workdir, shift=0, tma=True, order=0,
        fill=77, opt="-O0"):
    """Outputs {name: array} of one device call.  ``shift``: bytes from a
    256-byte boundary to the inputs' bases; ``fill``: the value outputs
    hold before the call; ``order``: 1 runs the threads of a CTA backwards
    between barriers."""
    from polymage_b200 import constructs as C
    from polymage_b200.evaluate import eval_int
    module = pipeline.generate_code()
    prms, ins, outs = pipeline.ordered_params()
    env = dict((p, int(params[p.name])) for p in prms
               if p.typ not in (C.Float, C.Double))
    dt = {C.Float: np.float32, C.Double: np.float64, C.Int: np.int32,
          C.UInt: np.uint32, C.Short: np.int16, C.UShort: np.uint16,
          C.Char: np.int8, C.UChar: np.uint8, C.Long: np.int64,
          C.ULong: np.uint64}
    bufs = []
    for f in ins + outs:
        shape = tuple(eval_int(d.upperBound - d.lowerBound + 1, env)
                      for d in f.domain)
        if f in ins:
            a = np.ascontiguousarray(inputs[f.name], dt[f.typ])
            assert a.shape == shape, (f.name, a.shape, shape)
        else:
            a = np.full(shape, fill, dt[f.typ])
        bufs.append(a)
    call = ", ".join(
        [("%rf" if p.typ in (C.Float, C.Double) else "%d") % (
            params[p.name],) for p in prms] +
        ["b[%d]" % i for i in range(len(bufs))] + ["nullptr"])
    write = "".join("fwrite(b[%d], 1, %d, f);" % (i, bufs[i].nbytes)
                    for i in range(len(ins), len(bufs)))
    src = _device_source(module.source) + \
        HOST.replace("EMU_NBUF", str(len(bufs))).replace(
            "EMU_CALL", "pipeline_%s_dev(%s)" % (module.name, call)).replace(
            "EMU_WRITE", write)
    os.makedirs(str(workdir), exist_ok=True)
    path = os.path.join(str(workdir), module.name)
    with open(path + ".cpp", "w") as f:
        f.write(src)
    srcs = [path + ".cpp"]
    if module.host_source:
        with open(path + "_host.cpp", "w") as f:
            f.write(module.host_source)
        srcs.append(path + "_host.cpp")
    r = subprocess.run(
        ["g++", opt, "-w", "-std=c++17", "-ffp-contract=off",
         "-fsanitize=address,bounds,alignment,null,shift-exponent",
         "-fno-sanitize-recover=all", "-I", CUDA_INC] + srcs +
        ["-o", path + ".exe", "-Wl,--unresolved-symbols=ignore-all"],
        stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
        universal_newlines=True)
    if r.returncode:
        raise EmulationError("g++:\n" + r.stdout[-6000:])
    with open(path + ".in", "wb") as f:
        for i, a in enumerate(bufs):
            f.write(np.array([a.nbytes, shift if i < len(ins) else 0],
                             np.int64).tobytes() + a.tobytes())
    e = dict(os.environ, EMU_ORDER=str(order),
             PM_DISABLE_TMA="0" if tma else "1",
             ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    r = subprocess.run([path + ".exe", path + ".in", path + ".out"], env=e,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       universal_newlines=True, timeout=600)
    if r.returncode:
        raise EmulationError("exit code %d\n%s" % (r.returncode,
                                                  r.stdout[:4000]))
    raw = np.fromfile(path + ".out", np.uint8)
    out, at = {}, 0
    for f, a in list(zip(ins + outs, bufs))[len(ins):]:
        out[f.name] = raw[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
        at += a.nbytes
    return out
