// Run-time compilation of fused elementwise tapes.
//
// The interpreter in k_map.cu runs any tape but pays for decoding and for keeping every value in
// shared memory: a chain of a dozen operations is bound by instruction issue at well under half
// of the HBM roofline.  Here the same SSA tape is written out as the body of a CUDA kernel,
// compiled for sm_100a with NVRTC, loaded through the driver API and cached by its text; values
// live in registers and the kernel is bound by HBM like the hand-written chain kernel.
//
// Same arithmetic as the interpreter, operation by operation: additions, subtractions and
// multiplications are emitted as __fadd_rn / __fsub_rn / __fmul_rn so that the compiler cannot
// contract two tape operations into one fused multiply-add, fused multiply-adds appear only where
// the tape says so, and the transcendental primitives are the same functions (tape_math.cuh is
// compiled into both).  The two paths therefore produce the same bits.
//
// The tape's constants are no part of the kernel unless the tape says that they never change (VRHI_TAPE_FLAG_LITERALS): they are
// passed by value at each launch, so two tapes that differ in nothing else, such as the frames of a loop with a
// moving uniform, share one kernel.
//
// NVRTC and the driver entry points are looked up at run time (dlopen, cudaGetDriverEntryPoint):
// the library neither links against them nor needs them unless a tape is launched.  Where NVRTC is
// not installed the interpreter runs instead; VRHI_TAPE_JIT=0 in the environment, or
// VRHI_TAPE_FLAG_INTERPRET in the parameter block, selects the interpreter explicitly.
#include <cuda.h>
#include <dlfcn.h>
#include <nvrtc.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "vrhi_internal.h"

namespace vrhi {

namespace {

const char kMathSource[] =
#include "tape_math_src.inc"
    ;

struct Nvrtc {
  decltype(&nvrtcCreateProgram) create = nullptr;
  decltype(&nvrtcCompileProgram) compile = nullptr;
  decltype(&nvrtcGetCUBINSize) cubin_size = nullptr;
  decltype(&nvrtcGetCUBIN) cubin = nullptr;
  decltype(&nvrtcGetProgramLogSize) log_size = nullptr;
  decltype(&nvrtcGetProgramLog) log = nullptr;
  decltype(&nvrtcDestroyProgram) destroy = nullptr;
  decltype(&nvrtcGetErrorString) error_string = nullptr;
  decltype(&nvrtcVersion) version = nullptr;
  int version_number = 0;  // major * 1000 + minor * 10, as CUDART_VERSION counts
  bool ok = false;
};

struct Driver {
  CUresult (*module_load_data)(CUmodule *, const void *) = nullptr;
  CUresult (*module_get_function)(CUfunction *, CUmodule, const char *) = nullptr;
  CUresult (*launch_kernel)(const CUlaunchConfig *, CUfunction, void **, void **) = nullptr;
  CUresult (*get_error_string)(CUresult, const char **) = nullptr;
  CUresult (*occupancy)(int *, CUfunction, int, size_t) = nullptr;
  bool ok = false;
};

std::mutex g_mu;
Nvrtc g_nvrtc;
Driver g_driver;
bool g_loaded = false;
uint64_t g_compiled = 0, g_launches = 0;
struct Compiled {
  CUfunction fn;
  int resident;  // blocks of 256 threads that fit on one SM at a time
};
std::unordered_map<std::string, Compiled> g_cache;  // key: device ordinal + the tape's description

template <class F>
bool sym(void *lib, const char *name, F *out) {
  *out = reinterpret_cast<F>(dlsym(lib, name));
  return *out != nullptr;
}

template <class F>
bool drv(const char *name, F *out) {
  void *p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess || !p) {
    (void)cudaGetLastError();
    return false;
  }
  *out = reinterpret_cast<F>(p);
  return true;
}

bool bind(void *lib, Nvrtc *out) {
  Nvrtc n;
  n.ok = sym(lib, "nvrtcCreateProgram", &n.create) && sym(lib, "nvrtcCompileProgram", &n.compile) &&
         sym(lib, "nvrtcGetCUBINSize", &n.cubin_size) && sym(lib, "nvrtcGetCUBIN", &n.cubin) &&
         sym(lib, "nvrtcGetProgramLogSize", &n.log_size) && sym(lib, "nvrtcGetProgramLog", &n.log) &&
         sym(lib, "nvrtcDestroyProgram", &n.destroy) && sym(lib, "nvrtcGetErrorString", &n.error_string) &&
         sym(lib, "nvrtcVersion", &n.version);
  if (!n.ok) return false;
  int major = 0, minor = 0;
  if (n.version(&major, &minor) != NVRTC_SUCCESS) return false;
  n.version_number = major * 1000 + minor * 10;
  *out = n;
  return true;
}

void load_once() {
  if (g_loaded) return;
  g_loaded = true;
  // The compiler whose version is the one this library was built with is preferred: its math
  // library is then the one the interpreting kernel was compiled against, which is what makes the
  // two paths agree bit for bit.  Any other NVRTC 12 still gives a correct kernel.
  const char *names[] = {getenv("VRHI_NVRTC"), "/usr/local/cuda/lib64/libnvrtc.so.12", "libnvrtc.so.12", "libnvrtc.so"};
  Nvrtc fallback;
  for (const char *name : names) {
    if (!name || !*name) continue;
    void *lib = dlopen(name, RTLD_NOW | RTLD_LOCAL);
    Nvrtc n;
    if (!lib || !bind(lib, &n)) continue;
    if (n.version_number / 10 == CUDART_VERSION / 10) { g_nvrtc = n; break; }
    if (!fallback.ok) fallback = n;
  }
  if (!g_nvrtc.ok && fallback.ok) g_nvrtc = fallback;
  Driver &d = g_driver;
  d.ok = drv("cuModuleLoadData", &d.module_load_data) && drv("cuModuleGetFunction", &d.module_get_function) &&
         drv("cuLaunchKernelEx", &d.launch_kernel) && drv("cuGetErrorString", &d.get_error_string) &&
         drv("cuOccupancyMaxActiveBlocksPerMultiprocessor", &d.occupancy);
}

inline bool tape_literal(const vrhi_tape_params &q) { return (q.flags & VRHI_TAPE_FLAG_LITERALS) != 0; }

std::string v(unsigned k) { return "v" + std::to_string(k); }

// One SSA instruction as a C expression over the values v<k>; `constant` is the name of a constant's value.
std::string expression(const vrhi_tape_instr &I, const std::string &constant) {
  const std::string a = v(I.a), b = v(I.b), c = v(I.c);
  switch (I.op) {
    case VRHI_T_CONST: return constant;
    case VRHI_T_ADD: return "__fadd_rn(" + a + ", " + b + ")";
    case VRHI_T_SUB: return "__fsub_rn(" + a + ", " + b + ")";
    case VRHI_T_MUL: return "__fmul_rn(" + a + ", " + b + ")";
    case VRHI_T_DIV: return a + " / " + b;
    case VRHI_T_MAX: return "fmaxf(" + a + ", " + b + ")";
    case VRHI_T_MIN: return "fminf(" + a + ", " + b + ")";
    case VRHI_T_EQ: return "(" + a + " == " + b + " ? 1.f : 0.f)";
    case VRHI_T_FMA: return "fmaf(" + a + ", " + b + ", " + c + ")";
    case VRHI_T_NEG: return "-" + a;
    case VRHI_T_ABS: return "fabsf(" + a + ")";
    case VRHI_T_SQUARE: return "__fmul_rn(" + a + ", " + a + ")";
    case VRHI_T_RELU: return "fmaxf(" + a + ", 0.0f)";
    case VRHI_T_SIGN: return "((" + a + " > 0.f) ? 1.f : ((" + a + " < 0.f) ? -1.f : 0.f))";
    case VRHI_T_STEP: return "(" + a + " > 0.f ? 1.f : 0.f)";
    case VRHI_T_SQRT: return "sqrtf(" + a + ")";
    case VRHI_T_RSQRT: return "1.0f / sqrtf(" + a + ")";
    case VRHI_T_RECIP: return "1.0f / " + a;
    case VRHI_T_EXP: return "expf(" + a + ")";
    case VRHI_T_LOG: return "logf(" + a + ")";
    case VRHI_T_TANH: return "tanhf(" + a + ")";
    case VRHI_T_SIGMOID: return "sigmoid_accurate(" + a + ")";
    case VRHI_T_COS: return "cosf(" + a + ")";
    default: return "sinf(" + a + ")";  // VRHI_T_SIN
  }
}

// How a generated kernel walks its arrays.  256 threads per block in both forms, float4 groups throughout.
//   FLAT    no row or column vectors, no column sums: one long array, grid-stride, whatever the row length; the up
//           to three elements behind the last float4 are done one by one by the first block.
//   ROWS    P = 4 / gcd(4, cols) rows together are a super row: P * cols elements, a multiple of 4, starting on a 16-byte
//           boundary.  A block owns a tile of W adjacent groups and takes R = 256 / W super rows at a time, thread t the
//           group t % W of the super rows t / W, t / W + R, ...: a narrow array keeps the whole block busy and neighbouring
//           threads read neighbouring addresses.  The four elements of a thread's group lie in the same columns in every super
//           row, so row vectors are loaded once per thread, and a partial row of column sums, one super row long, is P
//           partial rows of cols columns.  The rows % P rows behind the last super row are a partial one of `rem`
//           elements, done one by one by the thread that comes to it.  W and R are launch parameters.
// Measured on B200 against tiles of single elements for row lengths that are no multiple of 4: a tape over
// [1081,1919] 11.3 -> 8.2 us per call, a gradient graph of [2049,1001] 14.3 -> 12.4 us.
enum Form { FLAT, ROWS };

Form form_of(const vrhi_tape_params &q) {
  return (q.row_vector_mask | q.col_vector_mask | q.colsum_mask) == 0 ? FLAT : ROWS;
}
unsigned super_rows_of(uint64_t cols) { return cols % 4 == 0 ? 1 : cols % 2 == 0 ? 2 : 4; }

// `unroll` groups per thread and trip, the loads of all of them issued before any is used.  Row vectors and scalars are
// loaded once per thread, column vectors once per row.  An output is stored, or (colsum_mask) added up over the rows
// in a register, over the R rows of the block in shared memory, and written as one partial row per block row, or
// (total_mask) added up over everything the block visits and written as one partial value per block.
// `show_constants`: the values of this tape's constants as comments (they are no part of a compiled text).
std::string generate(const vrhi_tape_params &q, Form form, int unroll, bool show_constants = false) {
  const unsigned NI = q.n_inputs, NO = q.n_outputs, NT = q.n_instr;
  const unsigned P = super_rows_of(q.cols);
  const std::vector<std::string> comps{".x", ".y", ".z", ".w"};
  const std::string V = "float4", ULL = "unsigned long long";
  const std::string zero = "make_float4(0.f, 0.f, 0.f, 0.f)";
  auto splat = [&](const std::string &e) { return "make_float4(" + e + ", " + e + ", " + e + ", " + e + ")"; };
  auto str = [](unsigned k) { return std::to_string(k); };
  std::vector<bool> used(NI + NT, false);
  for (unsigned t = 0; t < NT; ++t) {
    const int ar = tape_arity(q.instr[t].op);
    const uint16_t src[3] = {q.instr[t].a, q.instr[t].b, q.instr[t].c};
    for (int s = 0; s < ar; ++s) used[src[s]] = true;
  }
  for (unsigned k = 0; k < NO; ++k) used[q.out_value[k]] = true;
  auto shape = [&](unsigned k) { return ((q.row_vector_mask >> k) & 1u) ? 'r' : ((q.col_vector_mask >> k) & 1u) ? 'c' : ((q.scalar_mask >> k) & 1u) ? 's' : 'f'; };
  auto colsum = [&](unsigned k) { return ((q.colsum_mask >> k) & 1u) != 0; };
  auto total = [&](unsigned k) { return tape_total(q, k); };
  bool any_colsum = false, any_total = false;
  for (unsigned k = 0; k < NO; ++k) { any_colsum = any_colsum || colsum(k); any_total = any_total || total(k); }

  const bool literal = tape_literal(q);
  unsigned NC = 0;
  for (unsigned t = 0; t < NT; ++t) NC += q.instr[t].op == VRHI_T_CONST && !literal;
  std::string constants;  // tape_body's arguments for them
  for (unsigned k = 0; k < NC; ++k) constants += "constants.k[" + str(k) + "], ";

  std::string s = kMathSource;
  if (NC) s += "\nstruct TapeConstants { float k[" + str(NC) + "]; };\n";
  s += "\n__device__ __forceinline__ void tape_body(";
  for (unsigned k = 0; k < NC; ++k) s += "const float k" + str(k) + ", ";
  for (unsigned k = 0; k < NI; ++k) s += "const float " + v(k) + ", ";
  for (unsigned k = 0; k < NO; ++k) s += "float &r" + str(k) + (k + 1 < NO ? ", " : "");
  s += ") {\n";
  for (unsigned t = 0, c = 0; t < NT; ++t) {
    const bool constant = q.instr[t].op == VRHI_T_CONST;
    uint32_t bits;
    memcpy(&bits, &q.instr[t].imm, 4);
    char value[48], comment[32];
    snprintf(value, sizeof value, "__int_as_float((int)0x%08xu)", bits);
    snprintf(comment, sizeof comment, "  // 0x%08x", bits);
    s += "  const float " + v(NI + t) + " = " + expression(q.instr[t], literal ? value : "k" + str(c)) + ";";
    if (constant && show_constants) s += comment;
    s += "\n";
    c += constant;
  }
  for (unsigned k = 0; k < NO; ++k) s += "  r" + str(k) + " = " + v(q.out_value[k]) + ";\n";
  s += "}\n\nextern \"C\" __global__ void __launch_bounds__(256) vrhi_tape_kernel(";
  for (unsigned k = 0; k < NI; ++k) s += "const float *__restrict__ in" + str(k) + ", ";
  for (unsigned k = 0; k < NO; ++k) s += "float *__restrict__ out" + str(k) + ", ";
  if (NC) s += "const __grid_constant__ TapeConstants constants, ";
  s += "const " + ULL + " rows, const " + ULL + " groups, const unsigned int W, const unsigned int R, const unsigned int tail, const " + ULL + " cols, const " + ULL + " rem, const unsigned int fold) {\n";
  s += "  asm volatile(\"griddepcontrol.wait;\" ::: \"memory\");  // a programmatic dependent of the kernel before it, and the next one of it\n  asm volatile(\"griddepcontrol.launch_dependents;\");\n";
  if (form == FLAT) {
    s += "  " + ULL + " i = (" + ULL + ")blockIdx.x * 256u + threadIdx.x;\n  const " + ULL + " step = (" + ULL + ")gridDim.x * 256u;\n";
  } else {
    s += "  const unsigned int sub = threadIdx.x / W, w = threadIdx.x - sub * W;\n";
    s += "  const " + ULL + " g = (" + ULL + ")blockIdx.x * W + w;\n  const bool active = sub < R && g < groups;\n";
    s += "  " + ULL + " row = (" + ULL + ")blockIdx.y * R + sub;\n  const " + ULL + " step = (" + ULL + ")gridDim.y * R, istep = step * groups;\n";
    s += "  " + ULL + " i = row * groups + g;\n";
    if (P > 1) {  // column and row (within the super row) of the group's four elements
      s += "  const " + ULL + " k0 = active ? 4ull * g : 0ull, r0 = (k0 >= cols) + (k0 >= 2ull * cols) + (k0 >= 3ull * cols), c0 = k0 - r0 * cols;\n";
      for (unsigned j = 1; j < 4; ++j)
        s += "  const " + ULL + " c" + str(j) + " = c" + str(j - 1) + " + 1ull == cols ? 0ull : c" + str(j - 1) + " + 1ull, r" + str(j) + " = r" + str(j - 1) + " + (c" + str(j) + " == 0ull);\n";
    }
  }
  for (unsigned k = 0; k < NI; ++k) {
    if (!used[k]) continue;
    const std::string K = str(k);
    if (shape(k) == 'r' && P > 1) s += "  const float4 x" + K + " = make_float4(__ldg(in" + K + " + c0), __ldg(in" + K + " + c1), __ldg(in" + K + " + c2), __ldg(in" + K + " + c3));\n";
    if (shape(k) == 'r' && P == 1) s += "  const " + V + " x" + K + " = active ? __ldg(reinterpret_cast<const " + V + " *>(in" + K + ") + g) : " + zero + ";\n";
    if (shape(k) == 's') s += "  const float s" + K + " = __ldg(in" + K + ");\n  const " + V + " x" + K + " = " + splat("s" + K) + ";\n";
  }
  for (unsigned k = 0; k < NO; ++k)
    if (colsum(k) || total(k)) s += "  " + V + " acc" + str(k) + " = " + zero + ";\n";
  // loads of one group, and its arithmetic and stores
  auto loads = [&](const std::string &G, const std::string &idx, const std::string &row) {
    std::string t;
    for (unsigned k = 0; k < NI; ++k) {
      if (!used[k]) continue;
      const std::string K = str(k), name = "x" + K + "_" + G;
      if (shape(k) == 'f') t += "      const " + V + " " + name + " = __ldcs(reinterpret_cast<const " + V + " *>(in" + K + ") + " + idx + ");\n";
      if (shape(k) == 'c' && P > 1) {
        t += "      const float *col" + K + "_" + G + " = in" + K + " + " + row + " * " + str(P) + "ull;\n      const float4 " + name + " = make_float4(";
        for (unsigned j = 0; j < 4; ++j) t += "__ldg(col" + K + "_" + G + " + r" + str(j) + (j < 3 ? "), " : "));\n");
      }
      if (shape(k) == 'c' && P == 1) t += "      const float c" + K + "_" + G + " = __ldg(in" + K + " + " + row + ");\n      const " + V + " " + name + " = " + splat("c" + K + "_" + G) + ";\n";
    }
    return t;
  };
  auto work = [&](const std::string &G, const std::string &idx) {
    std::string t = "      {\n";
    for (unsigned k = 0; k < NO; ++k) t += "        " + V + " o" + str(k) + ";\n";
    for (const std::string &c : comps) {
      t += "        tape_body(" + constants;
      for (unsigned k = 0; k < NI; ++k) {
        const std::string K = str(k);
        if (!used[k]) t += "0.0f, ";
        else if (shape(k) == 'r' || shape(k) == 's') t += "x" + K + c + ", ";
        else t += "x" + K + "_" + G + c + ", ";
      }
      for (unsigned k = 0; k < NO; ++k) t += "o" + str(k) + c + (k + 1 < NO ? ", " : "");
      t += ");\n";
    }
    for (unsigned k = 0; k < NO; ++k) {
      const std::string K = str(k);
      if (colsum(k) || total(k)) {  // groups are visited in a fixed order: the sum does not depend on scheduling
        t += "       ";
        for (const std::string &c : comps) t += " acc" + K + c + " += o" + K + c + ";";
        t += "\n";
      } else {
        t += "        __stcs(reinterpret_cast<" + V + " *>(out" + K + ") + " + idx + ", o" + K + ");\n";
      }
    }
    return t + "      }\n";
  };
  const std::string U = str((unsigned)unroll), last = str((unsigned)unroll - 1);
  const std::string advance = form == FLAT ? "i += " + U + "ull * step" : "row += " + U + "ull * step, i += " + U + "ull * istep";
  const std::string pos = form == FLAT ? "i" : "row", most = form == FLAT ? "groups" : "rows", di = form == FLAT ? "step" : "istep";
  if (form != FLAT) s += "  if (active) {\n";
  s += "  for (; " + pos + " + " + last + "ull * step < " + most + "; " + advance + ") {  // " + U + " complete groups per trip: all loads first\n";
  for (int k = 0; k < unroll; ++k) {
    const std::string G = str((unsigned)k);
    s += "      const " + ULL + " i" + G + " = i + " + G + "ull * " + di + (form == FLAT ? "" : ", row_" + G + " = row + " + G + "ull * step") + ";\n";
  }
  for (int k = 0; k < unroll; ++k) s += loads(str((unsigned)k), "i" + str((unsigned)k), "row_" + str((unsigned)k));
  for (int k = 0; k < unroll; ++k) s += work(str((unsigned)k), "i" + str((unsigned)k));
  s += "  }\n";
  s += "  for (; " + pos + " < " + most + "; " + (form == FLAT ? "i += step" : "row += step, i += istep") + ") {  // groups left over\n";
  s += loads("0", "i", "row") + work("0", "i");
  s += "  }\n";
  if (form == ROWS && P > 1) {  // the partial super row
    s += "  if (row == rows && 4ull * g < rem) {\n";
    for (unsigned j = 0; j < 4; ++j) {
      s += "    if (4ull * g + " + str(j) + "ull < rem) {\n      const " + ULL + " e = 4ull * i + " + str(j) + "ull;\n";
      for (unsigned k = 0; k < NO; ++k) s += "      float o" + str(k) + ";\n";
      s += "      tape_body(" + constants;
      for (unsigned k = 0; k < NI; ++k) {
        const std::string K = str(k);
        s += !used[k] ? std::string("0.0f") : shape(k) == 's' ? "s" + K : shape(k) == 'r' ? "x" + K + comps[j]
             : shape(k) == 'c' ? "__ldg(in" + K + " + row * " + str(P) + "ull + r" + str(j) + ")" : "in" + K + "[e]";
        s += ", ";
      }
      for (unsigned k = 0; k < NO; ++k) s += "o" + str(k) + (k + 1 < NO ? ", " : "");
      s += ");\n";
      for (unsigned k = 0; k < NO; ++k) s += colsum(k) || total(k) ? "      acc" + str(k) + comps[j] + " += o" + str(k) + ";\n" : "      out" + str(k) + "[e] = o" + str(k) + ";\n";
      s += "    }\n";
    }
    s += "  }\n";
  }
  if (form != FLAT) s += "  }\n";
  if (form == FLAT) {  // the elements behind the last float4
    s += "  if (blockIdx.x == 0 && threadIdx.x < tail) {\n      const " + ULL + " e = 4ull * groups + threadIdx.x;\n";
    for (unsigned k = 0; k < NO; ++k) s += "      float o" + str(k) + ";\n";
    s += "      tape_body(" + constants;
    for (unsigned k = 0; k < NI; ++k) s += !used[k] ? std::string("0.0f, ") : shape(k) == 's' ? "s" + str(k) + ", " : "in" + str(k) + "[e], ";
    for (unsigned k = 0; k < NO; ++k) s += "o" + str(k) + (k + 1 < NO ? ", " : "");
    s += ");\n";
    for (unsigned k = 0; k < NO; ++k) s += total(k) ? "      acc" + str(k) + ".x += o" + str(k) + ";\n" : "      out" + str(k) + "[e] = o" + str(k) + ";\n";
    s += "  }\n";
  }
  // column-summed outputs: a tree over the block's R rows, then this block row's partial super row, [gridDim.y][groups]
  if (any_colsum) s += "  __shared__ " + V + " red[256];\n";
  for (unsigned k = 0; k < NO; ++k) {
    if (!colsum(k)) continue;
    const std::string K = str(k);
    s += "  if (R > 1) {\n    __syncthreads();\n    red[threadIdx.x] = acc" + K + ";\n    for (unsigned int n = R; n > 1;) {\n      const unsigned int half = (n + 1) >> 1;\n      __syncthreads();\n";
    s += "      if (active && sub < n - half) {\n        const " + V + " other = red[threadIdx.x + half * W];\n       ";
    for (const std::string &c : comps) s += " acc" + K + c + " += other" + c + ";";
    s += "\n        red[threadIdx.x] = acc" + K + ";\n      }\n      n = half;\n    }\n  }\n";
    if (P > 1) {  // a block that holds whole super rows adds their rows up itself
      s += "  if (fold > 1) {\n    __syncthreads();\n    if (active && sub == 0) red[w] = acc" + K + ";\n    __syncthreads();\n    const float *sums = reinterpret_cast<const float *>(red);\n";
      s += "    for (unsigned int c = threadIdx.x; c < cols; c += 256u) {\n      float v = sums[c];\n      for (unsigned int k = 1; k < fold; ++k) v += sums[c + k * (unsigned int)cols];\n";
      s += "      out" + K + "[blockIdx.y * cols + c] = v;\n    }\n  } else\n";
    }
    s += "  if (active && sub == 0) reinterpret_cast<" + V + " *>(out" + K + ")[(" + ULL + ")blockIdx.y * groups + g] = acc" + K + ";\n";
  }
  // summed outputs: one partial value per block
  if (any_total) s += "  __shared__ float warp_total[8];\n";
  for (unsigned k = 0; k < NO; ++k) {
    if (!total(k)) continue;
    const std::string K = str(k);
    s += "  float t" + K + " = (acc" + K + ".x + acc" + K + ".y) + (acc" + K + ".z + acc" + K + ".w);\n";
    s += "  for (int o = 16; o > 0; o >>= 1) t" + K + " += __shfl_xor_sync(0xffffffffu, t" + K + ", o);\n";
    s += "  __syncthreads();\n  if ((threadIdx.x & 31u) == 0) warp_total[threadIdx.x >> 5] = t" + K + ";\n  __syncthreads();\n";
    s += "  if (threadIdx.x == 0) {\n    float t = warp_total[0];\n    for (int j = 1; j < 8; ++j) t += warp_total[j];\n    out" + K + "[(" + ULL + ")blockIdx.y * gridDim.x + blockIdx.x] = t;\n  }\n";
  }
  s += "}\n";
  return s;
}

int compile(vrhi_device_t *dev, const std::string &src, CUfunction *out) {
  nvrtcProgram prog = nullptr;
  nvrtcResult r = g_nvrtc.create(&prog, src.c_str(), "vrhi_tape.cu", 0, nullptr, nullptr);
  if (r != NVRTC_SUCCESS) return fail(VRHI_ERR_CUDA, "nvrtcCreateProgram: %s", g_nvrtc.error_string(r));
  char arch[64];
  snprintf(arch, sizeof arch, "--gpu-architecture=sm_%d%d%s", dev->prop.major, dev->prop.minor, dev->prop.major >= 9 ? "a" : "");
  const char *opts[] = {arch, "--std=c++17", "-lineinfo"};
  r = g_nvrtc.compile(prog, 3, opts);
  if (r != NVRTC_SUCCESS) {
    size_t n = 0;
    g_nvrtc.log_size(prog, &n);
    std::string log(n ? n : 1, '\0');
    if (n) g_nvrtc.log(prog, &log[0]);
    g_nvrtc.destroy(&prog);
    return fail(VRHI_ERR_CUDA, "compiling a fused tape failed: %s\n%.1500s", g_nvrtc.error_string(r), log.c_str());
  }
  size_t bytes = 0;
  g_nvrtc.cubin_size(prog, &bytes);
  std::vector<char> image(bytes);
  r = g_nvrtc.cubin(prog, image.data());
  g_nvrtc.destroy(&prog);
  if (r != NVRTC_SUCCESS || bytes == 0) return fail(VRHI_ERR_CUDA, "nvrtcGetCUBIN: %s", g_nvrtc.error_string(r));
  CUmodule mod = nullptr;
  CUresult cr = g_driver.module_load_data(&mod, image.data());
  const char *msg = "?";
  if (cr != CUDA_SUCCESS) {
    g_driver.get_error_string(cr, &msg);
    return fail(VRHI_ERR_CUDA, "cuModuleLoadData: %s", msg);
  }
  cr = g_driver.module_get_function(out, mod, "vrhi_tape_kernel");
  if (cr != CUDA_SUCCESS) {
    g_driver.get_error_string(cr, &msg);
    return fail(VRHI_ERR_CUDA, "cuModuleGetFunction: %s", msg);
  }
  return VRHI_OK;  // the module stays loaded for the life of the process (it is in the cache)
}

}  // namespace

// VRHI_TAPE_JIT=0 in the environment selects the interpreting kernel for every tape; read once per process
static bool jit_enabled() {
  static const bool on = env_int("VRHI_TAPE_JIT", 0, 1, 1) != 0;
  return on;
}

// Rows in flight per thread: about three 16-byte loads (measured on B200 with the three-input chain, 6.8 TB/s).
static int unroll_of(const vrhi_tape_params &q) {
  static const int env_unroll = env_int("VRHI_TAPE_UNROLL", 1, 8, 0);  // tuning aid
  if (env_unroll) return env_unroll;
  int full_inputs = 0;
  for (uint32_t k = 0; k < q.n_inputs; ++k)
    if (!(((q.row_vector_mask | q.col_vector_mask | q.scalar_mask) >> k) & 1u)) ++full_inputs;
  return full_inputs >= 3 ? 1 : full_inputs == 2 ? 2 : 3;
}

// The kernel of a tape, compiled if it is not there yet and the caller may wait for that; else 1.  g_mu is held.
static int find_kernel(vrhi_device_t *dev, const vrhi_tape_params &q, bool may_compile, Compiled *out) {
  const Form form = form_of(q);
  const int unroll = unroll_of(q);
  // cache key: everything the generated text depends on, as raw bytes (the text itself is only built on a miss).  The values
  // of constants are among it only where the tape says so.
  const bool literal = tape_literal(q);
  std::string key;
  const unsigned P = form == ROWS ? super_rows_of(q.cols) : 1u;
  const uint32_t head[13] = {(uint32_t)dev->ordinal, (uint32_t)unroll, (uint32_t)form, P, q.n_inputs, q.n_outputs, q.n_instr,
                             q.row_vector_mask, q.col_vector_mask, q.scalar_mask, q.colsum_mask, q.total_mask, literal};
  key.append(reinterpret_cast<const char *>(head), sizeof head);
  key.append(reinterpret_cast<const char *>(q.out_value), sizeof(uint32_t) * q.n_outputs);
  for (uint32_t t = 0; t < q.n_instr; ++t) {  // field by field: padding bytes of the struct are not defined
    const vrhi_tape_instr &I = q.instr[t];
    const uint16_t f[4] = {I.op, I.a, I.b, I.c};
    key.append(reinterpret_cast<const char *>(f), sizeof f);
    if (literal) key.append(reinterpret_cast<const char *>(&I.imm), sizeof I.imm);
  }
  auto it = g_cache.find(key);
  if (it == g_cache.end()) {
    if (!may_compile) return 1;
    VRHI_CUDA(cudaFree(nullptr));  // makes the device's primary context current for the driver calls below
    CUfunction fn = nullptr;
    VRHI_TRY(compile(dev, generate(q, form, unroll), &fn));
    int resident = 0;
    if (g_driver.occupancy(&resident, fn, 256, 0) != CUDA_SUCCESS || resident < 1) resident = 4;
    it = g_cache.emplace(key, Compiled{fn, resident}).first;
    ++g_compiled;
  }
  *out = it->second;
  return VRHI_OK;
}

int tape_jit_prepare(vrhi_device_t *dev, const vrhi_tape_params &q) {
  VRHI_CUDA(cudaSetDevice(dev->ordinal));
  std::lock_guard<std::mutex> lock(g_mu);
  load_once();
  if (!g_nvrtc.ok || !g_driver.ok) return VRHI_OK;
  Compiled unused;
  return find_kernel(dev, q, true, &unused);
}

// Returns VRHI_OK when the compiled kernel was launched, 1 when this tape or shape is left to the
// interpreter (no NVRTC, switched off, unaligned pointers, a handful of elements), and an error code when
// compilation or the launch failed.
int tape_jit_launch(vrhi_stream_t *st, const vrhi_tape_params &q, const float *const *in, float *const *out) {
  if (q.flags & VRHI_TAPE_FLAG_INTERPRET) return 1;
  if (!jit_enabled()) return 1;
  const Form form = form_of(q);
  const uint64_t n = q.rows * q.cols;
  // A few hundred elements take the time of a launch either way, and compiling costs a tenth of a second once.
  if (q.cols % 4 != 0 && n < 256 && !(q.colsum_mask | q.total_mask)) return 1;
  for (uint32_t k = 0; k < q.n_inputs; ++k)
    if (!((q.col_vector_mask >> k) & 1u) && !((q.scalar_mask >> k) & 1u) && ((uintptr_t)in[k] % 16)) return 1;
  for (uint32_t k = 0; k < q.n_outputs; ++k)
    if ((uintptr_t)out[k] % 16) return 1;

  std::lock_guard<std::mutex> lock(g_mu);
  load_once();
  if (!g_nvrtc.ok || !g_driver.ok) return 1;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  Compiled kernel;
  int rc = find_kernel(st->dev, q, false, &kernel);
  if (rc == 1) {
    VRHI_CUDA(cudaStreamIsCapturing(st->s, &cap));
    // a recording cannot wait for the compiler; what the interpreting kernel can do it does, with the same bits
    if (cap != cudaStreamCaptureStatusNone && !(q.colsum_mask | q.total_mask)) return 1;
    if (cap != cudaStreamCaptureStatusNone)
      return fail(VRHI_ERR_INVALID, "this tape has not been compiled yet; run the operator once on the stream before recording it");
    rc = find_kernel(st->dev, q, true, &kernel);
  }
  if (rc != VRHI_OK) return rc;
  struct { float k[VRHI_TAPE_MAX_INSTR]; } constants;
  uint32_t n_constants = 0;
  for (uint32_t t = 0; t < q.n_instr; ++t)
    if (q.instr[t].op == VRHI_T_CONST && !tape_literal(q)) constants.k[n_constants++] = q.instr[t].imm;
  // Six blocks per SM, all resident at once (one wave): measured on B200 with the three-input chain, eight blocks
  // per SM spill into a second, partly filled wave and two rows per trip then cost 15 %.
  static const int env_blocks = env_int("VRHI_TAPE_BLOCKS_PER_SM", 1, 32, 0);  // tuning aid
  const int unroll = unroll_of(q);
  const int most_blocks = 6;
  const uint64_t blocks_per_sm = env_blocks ? env_blocks : kernel.resident < most_blocks ? kernel.resident : most_blocks;
  const uint64_t target = (uint64_t)st->dev->prop.multiProcessorCount * blocks_per_sm;
  const unsigned P = form == ROWS ? super_rows_of(q.cols) : 1u;
  uint64_t rows = q.rows / P, groups, gx, gy = 1, cols = q.cols, rem = q.rows % P * q.cols;
  uint32_t W = 256, R = 1, tail = 0, fold = 1;
  if (form == FLAT) {
    groups = n / 4;
    tail = (uint32_t)(n % 4);
    gx = (groups + 255) / 256;
    if (gx > target) gx = target;
    if (gx == 0) gx = 1;
  } else {
    groups = P * q.cols / 4;
    // with column sums, tiles of 1 KiB: several super rows per block, so fewer partial rows
    const uint64_t most_w = q.colsum_mask ? 64 : 256;
    gx = (groups + most_w - 1) / most_w;
    if (gx > 0x7fffffffull) return fail(VRHI_ERR_UNSUPPORTED, "map_tape: too many columns");
    W = (uint32_t)((groups + gx - 1) / gx);
    R = 256u / W;
    if (gx == 1) fold = P;
    gy = target / gx;
    const uint64_t by_rows = (rows + (rem != 0) + (uint64_t)R * unroll - 1) / ((uint64_t)R * unroll);
    if (gy > by_rows) gy = by_rows;
    if (gy > 65535) gy = 65535;
    if (gy == 0) gy = 1;
  }
  void *args[VRHI_TAPE_MAX_INPUTS + VRHI_TAPE_MAX_OUTPUTS + 9];
  const float *in_copy[VRHI_TAPE_MAX_INPUTS];
  float *out_copy[VRHI_TAPE_MAX_OUTPUTS];
  int n_args = 0;
  for (uint32_t k = 0; k < q.n_inputs; ++k) { in_copy[k] = in[k]; args[n_args++] = &in_copy[k]; }
  FinishJobs jobs{};
  if (form == FLAT && q.total_mask && (q.rows == 1 || q.cols == 1) && !st->arena) {
    // Sums of a vector on a stream without scratch.  A recording cannot allocate it: one block, as row_sum has for a vector,
    // leaves its sum where the result goes.
    VRHI_CUDA(cudaStreamIsCapturing(st->s, &cap));
    if (cap != cudaStreamCaptureStatusNone) gx = gy = 1;
  }
  if (q.total_mask && !q.colsum_mask && gx * gy == 1) {
    for (uint32_t k = 0; k < q.n_outputs; ++k) {
      out_copy[k] = out[k];
      if (tape_total(q, k)) add_finish_job(&jobs, out[k], out[k], 1, 1, tape_mean(q, k) ? 1.0 / (double)n : 1.0);
    }
  } else if (q.colsum_mask | q.total_mask) {
    const size_t colsum_floats = (size_t)gy * P / fold * q.cols, total_floats = ((size_t)gx * gy + 3) & ~size_t(3);
    size_t floats = 0;
    for (uint32_t k = 0; k < q.n_outputs; ++k) floats += ((q.colsum_mask >> k) & 1u) ? (colsum_floats + 3) & ~size_t(3) : tape_total(q, k) ? total_floats : 0;
    char *scratch = nullptr;
    VRHI_TRY(stream_arena(st, floats * sizeof(float), nullptr, &scratch));
    float *next = reinterpret_cast<float *>(scratch);
    for (uint32_t k = 0; k < q.n_outputs; ++k) {
      out_copy[k] = out[k];
      if ((q.colsum_mask >> k) & 1u) {
        out_copy[k] = next;
        next += (colsum_floats + 3) & ~size_t(3);
        add_finish_job(&jobs, out_copy[k], out[k], (uint32_t)(gy * P / fold), q.cols, 1.0);
      } else if (tape_total(q, k)) {
        out_copy[k] = next;
        next += total_floats;
        add_finish_job(&jobs, out_copy[k], out[k], (uint32_t)(gx * gy), 1, tape_mean(q, k) ? 1.0 / (double)n : 1.0);
      }
    }
  } else {
    for (uint32_t k = 0; k < q.n_outputs; ++k) out_copy[k] = out[k];
  }
  for (uint32_t k = 0; k < q.n_outputs; ++k) args[n_args++] = &out_copy[k];
  if (n_constants) args[n_args++] = &constants;
  args[n_args++] = &rows; args[n_args++] = &groups; args[n_args++] = &W; args[n_args++] = &R; args[n_args++] = &tail; args[n_args++] = &cols; args[n_args++] = &rem; args[n_args++] = &fold;
  CUlaunchAttribute attr{};
  attr.id = CU_LAUNCH_ATTRIBUTE_PROGRAMMATIC_STREAM_SERIALIZATION;
  attr.value.programmaticStreamSerializationAllowed = 1;
  CUlaunchConfig cfg{};
  cfg.gridDimX = (unsigned)gx; cfg.gridDimY = (unsigned)gy; cfg.gridDimZ = 1;
  cfg.blockDimX = 256; cfg.blockDimY = 1; cfg.blockDimZ = 1;
  cfg.hStream = reinterpret_cast<CUstream>(st->s);
  cfg.attrs = &attr;
  cfg.numAttrs = chains(st) ? 1 : 0;
  CUresult cr = g_driver.launch_kernel(&cfg, kernel.fn, args, nullptr);
  if (cr != CUDA_SUCCESS) {
    const char *msg = "?";
    g_driver.get_error_string(cr, &msg);
    return fail(VRHI_ERR_CUDA, "launch of a compiled tape failed: %s", msg);
  }
  ++g_launches;
  if (jobs.n) {
    st->launches += 1;  // the tape's own kernel (the caller counts the last one)
    VRHI_CUDA(finish_partials(st->s, jobs));
  }
  return VRHI_OK;
}

bool tape_jit_available() {
  if (!jit_enabled()) return false;
  std::lock_guard<std::mutex> lock(g_mu);
  load_once();
  return g_nvrtc.ok && g_driver.ok;
}

void tape_jit_counters(uint64_t *compiled, uint64_t *launches, int *compiler_version, int *built_version) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (compiled) *compiled = g_compiled;
  if (launches) *launches = g_launches;
  if (compiler_version) *compiler_version = g_nvrtc.ok ? g_nvrtc.version_number : 0;
  if (built_version) *built_version = CUDART_VERSION / 10 * 10;
}

// The generated source of a tape, for inspection and for tests that run without a GPU.
std::string tape_jit_source(const vrhi_tape_params &q) {
  return generate(q, form_of(q), 2, true);
}

}  // namespace vrhi
