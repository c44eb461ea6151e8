// Host-level array operations: the counterparts of cuTile.jl's `ct.Tiled` broadcast (src/broadcast.jl: a whole
// broadcast expression fused into one kernel) and mapreduce (src/mapreduce.jl: sum / prod / maximum / minimum / a
// mapped reduction over any set of dimensions).  The reference compiles the Julia expression; a prebuilt library
// cannot, so the expression arrives as a short postfix program (push input, push constant, unary function, binary
// operator).  The host turns it into words of an accumulator machine with up to four temporaries (lower_program below:
// a leaf operand of a binary operator is read in place, constants and signs ride on other words, a value that occurs
// more than once is computed once), and every thread runs those words on registers for eight or sixteen elements at a time:
// still one pass over memory, one kernel, whatever the expression.  Arrays have up to three dimensions, column-major, first
// dimension contiguous; an operand with extent 1 along a dimension is expanded along it (stride 0).  Arithmetic is f32
// whatever the element type.  Both are bound by HBM bandwidth (bytes of the operands read once plus the result) as long as
// the expression is short.
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <optional>
#include <type_traits>

#include "ctx.h"
#include "ptx.cuh"

using namespace ctb_internal;

namespace {

constexpr int kMaxOps = CTB_TILED_MAX_OPS;
constexpr int kMaxInputs = CTB_TILED_MAX_INPUTS;
constexpr int kMaxConsts = CTB_TILED_MAX_CONSTS;
constexpr int kStack = 4;

// One instruction word of the accumulator machine.  The accumulator A is the top of a four-entry stack.
//   kind LOAD : push; A = operand
//   kind UNARY: A = code(A)
//   kind BIN  : A = A code operand, or operand code A when the REV bit is set; an operand from the stack is popped
// operand source: the stack entry below A (BIN only), inputs[arg] or constants[arg].
// Bits 24..31 of a word repeat kind, source, reversed and code as one dense index.
enum : unsigned { K_LOAD = 0, K_UNARY = 1, K_BIN = 2, K_STORE = 3 };
enum : unsigned { SRC_STACK = 0, SRC_INPUT = 1, SRC_CONST = 2, SRC_TEMP = 3 };  // STORE, TEMP: shared subexpressions only
constexpr unsigned kRevBit = 1u << 4;
constexpr unsigned dispatch_index(unsigned kind, unsigned src, bool rev, unsigned code) {
  return kind == K_LOAD    ? (src == SRC_INPUT ? 0u : 1u)
         : kind == K_UNARY ? 2u + (code - CTB_TILED_NEG)
                           : 14u + 7u * ((src == SRC_INPUT ? 0u : src == SRC_CONST ? 1u : 2u) * 2u + (rev ? 1u : 0u)) +
                                 (code - CTB_TILED_ADD);
}
constexpr unsigned make_ins(unsigned kind, unsigned src, bool rev, unsigned code, unsigned arg) {
  return kind | (src << 2) | (rev ? kRevBit : 0u) | (code << 8) | (arg << 16) | (dispatch_index(kind, src, rev, code) << 24);
}

// The kernel runs a lowered form without a stack: a value that waits (a stack entry, or a subexpression that occurs more
// than once) sits in one of up to kTemps temporaries.  A lowered word is operation | argument << 8 | tail bits: the result
// may still pass through A = p A + q (kTailFma) and be stored to temporary (word >> kTailStore) - 1 before the next word.
// What bounds long programs is the dispatch (about 24 issue slots and 200-400 clocks of latency per word and thread; the
// elements in flight are limited by registers), so words do much: adding, subtracting, multiplying by a constant and
// negation are one fused multiply-add with (p, q) chosen so that the result is the operator's own (A + c = 1 A + c,
// c - A = -1 A + c, A c = c A - 0, each rounded once) and ride on the word before them, subtracting an array is adding -1
// times it, and the eight operations that most expressions consist of are three compares deep behind one.
constexpr unsigned kSubtract = 1u << 10;    // L_ADD_*: A - operand
constexpr unsigned kOperandFma = 1u << 11;  // L_MUL_*, L_ADD_*: the operand enters as p operand + q
constexpr unsigned kTailFma = 1u << 12;
constexpr int kTailStore = 13;
enum : unsigned {
  L_FMA = 0,                                       // A = p A + q
  L_LOAD_INPUT, L_LOAD_TEMP,                       // A = operand
  L_MUL_INPUT, L_MUL_TEMP, L_ADD_INPUT, L_ADD_TEMP,  // A = A * operand, A +- operand
  L_LOAD_CONST,                                    // A = q
  L_HOT,                                           // number of the operations above
  L_UNARY = L_HOT,                                 // + code - NEG
  L_BINARY = L_UNARY + (CTB_TILED_ABS2 - CTB_TILED_NEG + 1),  // + 10 * source + 2 * (SUB, DIV, MAX, MIN, POW) + reversed
  L_COUNT = L_BINARY + 30
};
constexpr int kColdCodes[5] = {CTB_TILED_SUB, CTB_TILED_DIV, CTB_TILED_MAX, CTB_TILED_MIN, CTB_TILED_POW};
constexpr int kTemps = 4;
constexpr int kMaxIns = CTB_TILED_MAX_WORDS;  // a word per operation, and what the stores of temporaries add

struct Program {
  int n_ins;
  int n_temps;
  unsigned ins[kMaxIns + 1];  // one word of padding: the kernel fetches a word ahead
  float2 pq[kMaxIns];
  // Offset of the temporaries in shared memory.  Here and not among the operands, where four bytes more move the words and their
  // constants: f32 expressions without temporaries took 6 to 13 % longer (1000 x 1000, A + B: 3.6 us, then 4.0).
  unsigned temp_slot;
  bool operand_fma;  // some word has kOperandFma: the kernel without temporaries does not look for it
};

// How an operand is read (chosen on the host).
enum : int {
  OP_LINEAR = 0,  // laid out like the destination, aligned: a vector of four elements per group
  OP_SCALAR = 1,  // a single element
  OP_ROW = 2,     // expanded, first extent a multiple of four: one aligned vector per group
  OP_SHIFTED = 3, // laid out like the destination, not aligned: element by element
  OP_ELEM = 4,    // anything else: element by element, each with its own coordinates
  OP_VECTOR = 5,  // OP_ROW that varies along the first dimension only (a bias): one aligned vector per group
  OP_GROUP = 7,   // expanded along the first dimension, whose extent is a multiple of four: one element per group
  OP_FIXED = 6    // varies along the first dimension only, and the grid is such that every group of a thread lies at the
                  // same place of it: four elements per thread, read once
};
struct Operands {
  const void* ptr[kMaxInputs];
  long long stride[kMaxInputs][3];
  int mode[kMaxInputs];
  unsigned slot[kMaxInputs];  // offset in shared memory
};

// ---- postfix program -> accumulator-machine instructions (host) ---------------------------------------------------
struct Node {
  int op, arg, left, right;  // left/right: node indices, -1 for none
  int need;                  // stack entries the subtree needs when it is evaluated into A
  int uses, temp;            // times it is an operand; temporary that holds it once evaluated, -1 for none
};
inline bool is_input(const Node& n) { return n.op == CTB_TILED_INPUT; }

struct Compiler {
  Node nodes[kMaxOps];
  int n_nodes = 0, n_words = 0;
  bool lowering = false;
  const float* constants = nullptr;  // lowering only
  unsigned words[kMaxIns];           // with a stack; kind STORE only for shared subexpressions
  float2 affine[kMaxIns];            // of words with an operand p leaf + q, else (0, 0)
  void put(unsigned w) {
    affine[n_words] = make_float2(0.f, 0.f);
    words[n_words++] = w;
  }
  bool plain(int i) const { return nodes[i].op == CTB_TILED_INPUT || nodes[i].op == CTB_TILED_CONST || nodes[i].temp >= 0; }
  bool leaf(int i) const { return plain(i); }
  // Is node i = p leaf + q with one rounding, the leaf an input or a temporary?  Such an operand of + - * needs no
  // evaluation of its own when lowered.
  bool affine_leaf(int i, int* of, float* p, float* q) const {
    if (!lowering || plain(i)) return false;
    const Node& n = nodes[i];
    auto array = [&](int k) { return plain(k) && (nodes[k].temp >= 0 || nodes[k].op == CTB_TILED_INPUT); };
    if (n.op == CTB_TILED_NEG && array(n.left)) {
      *of = n.left; *p = -1.f; *q = -0.f;
      return true;
    }
    if (n.op < CTB_TILED_ADD || n.op > CTB_TILED_MUL) return false;
    const bool left = array(n.left);
    const int a = left ? n.left : n.right, k = left ? n.right : n.left;
    if (!array(a) || nodes[k].op != CTB_TILED_CONST) return false;
    const float v = constants[nodes[k].arg];
    *of = a;
    if (n.op == CTB_TILED_MUL) { *p = v; *q = -0.f; }
    else if (n.op == CTB_TILED_ADD) { *p = 1.f; *q = v; }
    else { *p = left ? 1.f : -1.f; *q = left ? -v : v; }
    return true;
  }
  unsigned leaf_src(int i) const { return nodes[i].temp >= 0 ? SRC_TEMP : is_input(nodes[i]) ? SRC_INPUT : SRC_CONST; }
  unsigned leaf_arg(int i) const { return (unsigned)(nodes[i].temp >= 0 ? nodes[i].temp : nodes[i].arg); }
  // stack entries of every node from those of its operands (operands come before their operators)
  void set_needs() {
    for (int i = 0; i < n_nodes; ++i) {
      Node& n = nodes[i];
      n.need = 1;
      if (n.left < 0) continue;
      const int l = leaf(n.left) ? 1 : nodes[n.left].need;
      if (n.right < 0) { n.need = l; continue; }
      const int r = leaf(n.right) ? 1 : nodes[n.right].need;
      int of;
      float p, q;
      const bool in_place = n.op <= CTB_TILED_MUL && !leaf(n.left) && !leaf(n.right);
      if (in_place && affine_leaf(n.right, &of, &p, &q)) { n.need = l; continue; }
      if (in_place && n.op != CTB_TILED_SUB && affine_leaf(n.left, &of, &p, &q)) { n.need = r; continue; }
      n.need = leaf(n.right) ? l : leaf(n.left) ? r : std::max(std::max(l, r), std::min(l, r) + 1);
    }
  }
  void emit(int i) {  // the value of a node (a leaf only when it is the whole expression) into A
    const Node& n = nodes[i];
    if (leaf(i)) {
      put(make_ins(K_LOAD, leaf_src(i), false, 0, leaf_arg(i)));
    } else {
      emit_op(i);
    }
  }
  void emit_op(int i) {
    const Node& n = nodes[i];
    if (n.right < 0) {
      emit(n.left);
      if (n.op != CTB_TILED_IDENTITY) put(make_ins(K_UNARY, 0, false, (unsigned)n.op, 0));
      return;
    }
    const bool commutes = n.op == CTB_TILED_ADD || n.op == CTB_TILED_MUL;  // a op b == b op a bit for bit
    int of;
    float p, q;
    if (n.op <= CTB_TILED_MUL && !leaf(n.left) && !leaf(n.right)) {
      const bool right = affine_leaf(n.right, &of, &p, &q);
      if (right || (commutes && affine_leaf(n.left, &of, &p, &q))) {  // A = one side; A = A op (p leaf + q)
        emit(right ? n.left : n.right);
        put(make_ins(K_BIN, leaf_src(of), false, (unsigned)n.op, leaf_arg(of)));
        affine[n_words - 1] = make_float2(p, q);
        return;
      }
    }
    if (leaf(n.right)) {        // A = left; A = A op leaf
      emit(n.left);
      put(make_ins(K_BIN, leaf_src(n.right), false, (unsigned)n.op, leaf_arg(n.right)));
    } else if (leaf(n.left)) {  // A = right; A = leaf op A
      emit(n.right);
      put(make_ins(K_BIN, leaf_src(n.left), !commutes, (unsigned)n.op, leaf_arg(n.left)));
    } else if (nodes[n.left].need > nodes[n.right].need) {  // the deeper side first: A = right, below it left; A = below op A
      emit(n.left);
      emit(n.right);
      put(make_ins(K_BIN, SRC_STACK, !commutes, (unsigned)n.op, 0));
    } else {                    // A = left, below it right; A = A op below
      emit(n.right);
      emit(n.left);
      put(make_ins(K_BIN, SRC_STACK, false, (unsigned)n.op, 0));
    }
  }
};

// Parses the postfix program into c (the root is the last node).  Returns 0, or a negative number -(k+1) naming the
// offending operation k with *why set.  share: equal subexpressions become one node (value numbering).
int parse_program(const int32_t* program, int n_ops, int n_inputs, int n_constants, bool share, Compiler* c, int* root,
                  const char** why) {
  int stack[kMaxOps], depth = 0;
  for (int k = 0; k < n_ops; ++k) {
    const int op = program[2 * k], arg = program[2 * k + 1];
    Node n = {op, 0, -1, -1, 1, 0, -1};
    if (op == CTB_TILED_INPUT) {
      if (arg < 0 || arg >= n_inputs) { *why = "names an input that was not given"; return -(k + 1); }
      n.arg = arg;
    } else if (op == CTB_TILED_CONST) {
      if (arg < 0 || arg >= n_constants) { *why = "names a constant that was not given"; return -(k + 1); }
      n.arg = arg;
    } else if (op >= CTB_TILED_IDENTITY && op <= CTB_TILED_ABS2) {
      if (depth < 1) { *why = "finds an empty stack"; return -(k + 1); }
      n.left = stack[--depth];
    } else if (op >= CTB_TILED_ADD && op <= CTB_TILED_POW) {
      if (depth < 2) { *why = "needs two values on the stack"; return -(k + 1); }
      n.right = stack[--depth];
      n.left = stack[--depth];
    } else {
      *why = "is not an operation code";
      return -(k + 1);
    }
    int at = c->n_nodes;
    if (share) {
      at = 0;
      auto same = [&](const Node& m) { return m.op == n.op && m.arg == n.arg && m.left == n.left && m.right == n.right; };
      while (at < c->n_nodes && !same(c->nodes[at])) ++at;
    }
    if (at == c->n_nodes) {
      if (n.left >= 0) ++c->nodes[n.left].uses;
      if (n.right >= 0) ++c->nodes[n.right].uses;
      c->nodes[c->n_nodes++] = n;
    }
    stack[depth++] = at;
  }
  if (depth != 1) { *why = "the program must leave exactly one value"; return -(n_ops + 1); }
  *root = stack[0];
  return 0;
}

// The instructions with a stack, without sharing (what ctb_tiled_compile reports); -1000 when the expression needs more
// than kStack live values.
int compile_program(const int32_t* program, int n_ops, int n_inputs, int n_constants, Compiler* c, const char** why) {
  int root;
  const int bad = parse_program(program, n_ops, n_inputs, n_constants, false, c, &root, why);
  if (bad) return bad;
  c->set_needs();
  if (c->nodes[root].need > kStack) return -1000;
  c->emit(root);
  return 0;
}

// The lowered program of the kernel.  Subexpressions that occur more than once are evaluated first, each into a temporary
// of its own (v = x + b is computed once in 0.5 v (1 + tanh(c (v + k v v v))): 11 instructions instead of 22), those that
// save most first, as far as the temporaries reach; the rest is evaluated where it occurs.
int lower_program(const int32_t* program, int n_ops, int n_inputs, const float* constants, int n_constants, Program* out,
                  const char** why) {
  Compiler c;
  c.lowering = true;
  c.constants = constants;
  int root;
  const int bad = parse_program(program, n_ops, n_inputs, n_constants, true, &c, &root, why);
  if (bad) return bad;
  int cost[kMaxOps];  // operators in the tree below a node
  for (int i = 0; i < c.n_nodes; ++i) {
    const Node& n = c.nodes[i];
    cost[i] = n.left < 0 ? 0 : 1 + cost[n.left] + (n.right < 0 ? 0 : cost[n.right]);
  }
  auto stack_need = [&]() {  // over the root and every shared subexpression
    c.set_needs();
    int need = c.nodes[root].need;
    for (int i = 0; i < c.n_nodes; ++i)
      if (c.nodes[i].temp >= 0) need = std::max(need, c.nodes[i].need);
    return need;
  };
  if (stack_need() > kStack) return -1000;
  int shared = 0;
  bool tried[kMaxOps] = {};
  for (;;) {
    int best = -1;
    for (int i = 0; i < c.n_nodes; ++i)
      if (!tried[i] && i != root && c.nodes[i].uses > 1 && cost[i] > 0 &&
          (best < 0 || cost[i] * (c.nodes[i].uses - 1) > cost[best] * (c.nodes[best].uses - 1)))
        best = i;
    if (best < 0) break;
    tried[best] = true;
    c.nodes[best].temp = 0;  // any value: the leaf test
    if (stack_need() - 1 + shared + 1 > kTemps) c.nodes[best].temp = -1;
    else ++shared;
  }
  int next = stack_need() - 1;  // stack entries take the first temporaries
  out->n_temps = next + shared;
  out->operand_fma = false;
  for (int i = 0; i < c.n_nodes; ++i)
    if (c.nodes[i].temp >= 0) c.nodes[i].temp = next++;
  for (int i = 0; i < c.n_nodes; ++i)
    if (c.nodes[i].temp >= 0) {
      c.emit_op(i);
      c.put(make_ins(K_STORE, 0, false, 0, (unsigned)c.nodes[i].temp));
    }
  c.emit(root);
  // stack -> temporaries: the value at depth d of the stack (0 = bottom) waits in temporary d
  out->n_ins = 0;
  int depth = 0, held = -1;  // held: the temporary whose value A holds as well, -1 for none
  bool tail_free = false;  // the last word can still take a multiply-add
  auto put = [&](unsigned op, unsigned arg, float q, bool uses_q) {
    out->pq[out->n_ins].x = 0.f;
    out->pq[out->n_ins].y = q;
    out->ins[out->n_ins++] = op | (arg << 8);
    held = -1;
    tail_free = !uses_q;
  };
  auto fma = [&](float p, float q) {  // A = p A + q
    if (!tail_free) put(L_FMA, 0, 0.f, true);
    else out->ins[out->n_ins - 1] |= kTailFma;
    out->pq[out->n_ins - 1].x = p;
    out->pq[out->n_ins - 1].y = q;
    tail_free = false;
    held = -1;
  };
  auto store = [&](int t) {  // with the word that computed the value
    if (out->ins[out->n_ins - 1] >> kTailStore) fma(1.f, -0.f);  // that one stores already: A = A
    out->ins[out->n_ins - 1] |= (unsigned)(t + 1) << kTailStore;
    tail_free = false;
    held = t;
  };
  for (int k = 0; k < c.n_words; ++k) {
    const unsigned w = c.words[k], kind = w & 3u, src = (w >> 2) & 3u, code = (w >> 8) & 0xffu, arg = (w >> 16) & 0xffu;
    const bool rev = (w & kRevBit) != 0;
    if (kind == K_LOAD) {
      if (depth > 0) store(depth - 1);
      ++depth;
      if (src == SRC_INPUT) put(L_LOAD_INPUT, arg, 0.f, false);
      else if (src == SRC_CONST) put(L_LOAD_CONST, 0, constants[arg], true);
      else if ((int)arg != held) put(L_LOAD_TEMP, arg, 0.f, false);
    } else if (kind == K_UNARY) {
      if (code == CTB_TILED_NEG) fma(-1.f, -0.f);
      else put(L_UNARY + code - CTB_TILED_NEG, 0, 0.f, false);
    } else if (kind == K_STORE) {
      store((int)arg);
      depth = 0;
    } else {
      unsigned from = src, index = arg;
      if (src == SRC_STACK) {
        --depth;
        from = SRC_TEMP;
        index = (unsigned)(depth - 1);
      }
      const bool in = from == SRC_INPUT;
      const float2 aff = c.affine[k];
      if (aff.x != 0.f || aff.y != 0.f || std::signbit(aff.y)) {
        put(code == CTB_TILED_MUL ? (in ? L_MUL_INPUT : L_MUL_TEMP) : (in ? L_ADD_INPUT : L_ADD_TEMP),
            index | (code == CTB_TILED_SUB ? kSubtract >> 8 : 0u) | kOperandFma >> 8, aff.y, true);
        out->pq[out->n_ins - 1].x = aff.x;
        out->operand_fma = true;
      } else if (from == SRC_CONST && code <= CTB_TILED_MUL) {
        const float v = constants[index];
        if (code == CTB_TILED_ADD) fma(1.f, v);
        else if (code == CTB_TILED_MUL) fma(v, -0.f);
        else if (rev) fma(-1.f, v);
        else fma(1.f, -v);
      } else if (code == CTB_TILED_MUL) {
        put(in ? L_MUL_INPUT : L_MUL_TEMP, index, 0.f, false);
      } else if (code == CTB_TILED_ADD || (code == CTB_TILED_SUB && !rev)) {
        put(in ? L_ADD_INPUT : L_ADD_TEMP, index | (code == CTB_TILED_ADD ? 0u : kSubtract >> 8), 0.f, false);
      } else {
        unsigned pos = 0;
        while (kColdCodes[pos] != (int)code) ++pos;
        put(L_BINARY + 10u * (in ? 0u : from == SRC_CONST ? 1u : 2u) + 2u * pos + (rev ? 1u : 0u), index,
            from == SRC_CONST ? constants[index] : 0.f, from == SRC_CONST);
      }
    }
  }
  return 0;
}

__device__ __forceinline__ float unary(int op, float x) {
  switch (op) {
    case CTB_TILED_NEG: return -x;
    case CTB_TILED_ABS: return fabsf(x);
    case CTB_TILED_SQRT: return sqrtf(x);
    case CTB_TILED_EXP: return expf(x);
    case CTB_TILED_EXP2: return exp2f(x);
    case CTB_TILED_LOG: return logf(x);
    case CTB_TILED_LOG2: return log2f(x);
    case CTB_TILED_SIN: return sinf(x);
    case CTB_TILED_COS: return cosf(x);
    case CTB_TILED_TANH: return tanhf(x);
    case CTB_TILED_INV: return 1.0f / x;
    case CTB_TILED_ABS2: return x * x;
    default: return x;  // CTB_TILED_IDENTITY
  }
}
__device__ __forceinline__ float binary(int op, float a, float b) {
  switch (op) {
    case CTB_TILED_ADD: return a + b;
    case CTB_TILED_SUB: return a - b;
    case CTB_TILED_MUL: return a * b;
    case CTB_TILED_DIV: return a / b;
    case CTB_TILED_MAX: return fmaxf(a, b);
    case CTB_TILED_MIN: return fminf(a, b);
    default: return powf(a, b);  // CTB_TILED_POW
  }
}

template <typename T>
__device__ __forceinline__ float load1(const void* p, long long i) {
  if constexpr (sizeof(T) == 4) return static_cast<const float*>(p)[i];
  else return __half2float(static_cast<const __half*>(p)[i]);
}
template <typename T>
__device__ __forceinline__ void store1(void* p, long long i, float v) {
  if constexpr (sizeof(T) == 4) static_cast<float*>(p)[i] = v;
  else static_cast<__half*>(p)[i] = __float2half_rn(v);
}

// ---- sine and cosine for the vector path ---------------------------------------------------------------------------
// The library's sinf / cosf test every element for a huge argument and branch; for a thread's 4 * G elements that
// is most of the instructions of a short expression.  Here the test is made once for all of a thread's elements and
// the common case runs without a branch:  j = round(|x| * 2/pi) by the magic-number addition, r = |x| - j * pi/2 with
// pi/2 split in three f32 parts (every step one FMA; for |x| <= 105615 the first difference is exact), then
// sin(r) = r + r s (S0 + S1 s + S2 s^2) or cos(r) = 1 - s/2 + s^2 (C0 + C1 s + C2 s^2) with s = r^2, picked by the
// parity of j, the sign by bit 1 of j (and by the sign of x for the sine, which keeps sin(-0) = -0).  The
// coefficients are a weighted minimax fit on |r| <= pi/4 (fit errors 3.6e-9 relative and 9.6e-11).  The same
// arithmetic evaluated on a CPU for every f32 in [0, 105615] differs from the exact value by at most 1.54 ulp
// (0.02 % of the arguments by more than 1 ulp).  Anything larger, infinite or NaN takes sinf / cosf.
constexpr float kSinCosLimit = 105615.0f;
template <bool COS>
__device__ __forceinline__ float sincos_reduced(float x) {
  constexpr float kTwoOverPi = 0.636619772367581343f, kMagic = 12582912.0f;  // 1.5 * 2^23
  constexpr float P1 = 0x1.921fb6p+0f, P2 = -0x1.777a5cp-25f, P3 = -0x1.ee59dap-50f;  // sum = pi/2 to 2^-74
  constexpr float S0 = -0.16666655242443085f, S1 = 0.008332176133990288f, S2 = -0.00019516977772582322f;
  constexpr float C0 = 0.04166664555668831f, C1 = -0.0013887364184483886f, C2 = 2.443809171381872e-05f;
  const float ax = fabsf(x);
  float jf = __fmaf_rn(ax, kTwoOverPi, kMagic);
  unsigned q = __float_as_uint(jf);  // the low bits of the mantissa hold j
  jf = __fadd_rn(jf, -kMagic);
  float r = __fmaf_rn(jf, -P1, ax);
  r = __fmaf_rn(jf, -P2, r);
  r = __fmaf_rn(jf, -P3, r);
  if (COS) q += 1u;  // cos(x) = sin(x + pi/2)
  const float s = __fmul_rn(r, r);
  // both polynomials, one select: selects and bit operations issue at half the rate of FMAs
  float ps = __fmaf_rn(s, S2, S1);
  ps = __fmaf_rn(s, ps, S0);
  ps = __fmaf_rn(__fmul_rn(s, r), ps, r);
  float pc = __fmaf_rn(s, C2, C1);
  pc = __fmaf_rn(s, pc, C0);
  pc = __fmaf_rn(s, pc, -0.5f);
  pc = __fmaf_rn(s, pc, 1.0f);
  const float res = (q & 1u) ? pc : ps;
  unsigned sign = (q & 2u) << 30;
  if (!COS) sign ^= __float_as_uint(x) & 0x80000000u;
  return __uint_as_float(__float_as_uint(res) ^ sign);
}
template <bool COS, int E>
__device__ __forceinline__ void sincos_all(float (&a)[E]) {
  bool in_range = true;
#pragma unroll
  for (int v = 0; v < E; ++v) in_range = in_range && (fabsf(a[v]) <= kSinCosLimit);  // false for NaN
  if (in_range) {
#pragma unroll
    for (int v = 0; v < E; ++v) a[v] = sincos_reduced<COS>(a[v]);
  } else {
#pragma unroll
    for (int v = 0; v < E; ++v) a[v] = COS ? cosf(a[v]) : sinf(a[v]);
  }
}

// ---- the kernel: operands staged in shared memory by cp.async, two trips deep ---------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// 16 or 8 bytes global -> shared, asynchronous; the bytes beyond src_bytes become zeros and are not read
template <int BYTES>
__device__ __forceinline__ void cp_async_group(unsigned dst, const void* src, unsigned src_bytes) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// one element global -> shared (asynchronous for 4-byte elements); zero when !live
template <typename T>
__device__ __forceinline__ void copy_element(unsigned dst, const T* src, bool live) {
  if constexpr (sizeof(T) == 4) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4u : 0u) : "memory");
  } else {
    const unsigned short v = live ? *reinterpret_cast<const unsigned short*>(src) : (unsigned short)0;
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst), "h"(v) : "memory");
  }
}

// A thread's values live in 64-bit registers of two neighbouring elements each: + and * then take half an instruction per
// element (with single floats in between, the moves into aligned register pairs and back cost more than the arithmetic).
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair(float lo, float hi) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpair(Pair p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ Pair fma_pair(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ Pair mul_pair(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The element-wise part of an instruction that is neither + nor *.  The operation, its direction and the
// kind of operand are template parameters and every instruction has its own straight-line code under the kernel's
// dispatch.
template <int CODE, bool REV>
__device__ __forceinline__ float binary_op(float p, float q) {
  const float a = REV ? q : p, b = REV ? p : q;
  if constexpr (CODE == CTB_TILED_SUB) return a - b;
  else if constexpr (CODE == CTB_TILED_DIV) return a / b;
  else if constexpr (CODE == CTB_TILED_MAX) return fmaxf(a, b);
  else if constexpr (CODE == CTB_TILED_MIN) return fminf(a, b);
  else return powf(a, b);
}
template <int CODE, bool REV, int H, typename Get>
__device__ __forceinline__ void apply_binary(Pair (&s0)[H], Get t) {  // t(h): the operand of pair h
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const float2 a = unpair(s0[h]), b = unpair(t(h));
    s0[h] = pair(binary_op<CODE, REV>(a.x, b.x), binary_op<CODE, REV>(a.y, b.y));
  }
}
// tanh of two elements.  The library's tanhf branches per element (20 instructions measured); here both forms are
// evaluated, the polynomials two elements at a time (12.5): |x| <= 1.25: x + x s P(s) with s = x^2 and P a weighted
// minimax fit of degree 7 (fit error 1.0e-8 relative), above: 1 - 2 / (e^(2|x|) + 1).  Evaluated in C with the errors
// that the exp2 and reciprocal units may add, the result is within 1.6 ulp everywhere.
__device__ __forceinline__ Pair tanh_pair(Pair x) {
  constexpr float kP[8] = {-0x1.555528p-2f, 0x1.110984p-3f, -0x1.b93bb2p-5f, 0x1.5fe566p-6f,
                           -0x1.077b52p-7f, 0x1.4a90acp-9f, -0x1.1f4f08p-11f, 0x1.e7bc34p-15f};
  constexpr float kTwoLog2e = 2.885390081777927f, kSwitch = 1.25f;
  const float2 xs = unpair(x);
  const float2 af = make_float2(fabsf(xs.x), fabsf(xs.y));
  const Pair a = pair(af.x, af.y), s = mul_pair(a, a);
  Pair poly = pair(kP[7], kP[7]);
#pragma unroll
  for (int k = 6; k >= 0; --k) poly = fma_pair(s, poly, pair(kP[k], kP[k]));
  poly = fma_pair(mul_pair(a, s), poly, a);
  const float2 t = unpair(mul_pair(a, pair(kTwoLog2e, kTwoLog2e)));
  const float2 e1 = make_float2(ctb::ex2_approx_ftz(t.x) + 1.f, ctb::ex2_approx_ftz(t.y) + 1.f);
  const Pair big = fma_pair(pair(ctb::rcp_approx_ftz(e1.x), ctb::rcp_approx_ftz(e1.y)), pair(-2.f, -2.f), pair(1.f, 1.f));
  const float2 ps = unpair(poly), bs = unpair(big);
  return pair(copysignf(af.x > kSwitch ? bs.x : ps.x, xs.x), copysignf(af.y > kSwitch ? bs.y : ps.y, xs.y));
}

template <int CODE, int H>
__device__ __forceinline__ void apply_unary(Pair (&s0)[H]) {
  if constexpr (CODE == CTB_TILED_TANH) {
#pragma unroll
    for (int h = 0; h < H; ++h) s0[h] = tanh_pair(s0[h]);
    return;
  }
  float f[2 * H];
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const float2 a = unpair(s0[h]);
    f[2 * h] = a.x;
    f[2 * h + 1] = a.y;
  }
  if constexpr (CODE == CTB_TILED_SIN) {
    sincos_all<false>(f);
  } else if constexpr (CODE == CTB_TILED_COS) {
    sincos_all<true>(f);
  } else {
#pragma unroll
    for (int v = 0; v < 2 * H; ++v) f[v] = unary(CODE, f[v]);  // CODE is a constant: the switch inside folds
  }
#pragma unroll
  for (int h = 0; h < H; ++h) s0[h] = pair(f[2 * h], f[2 * h + 1]);
}

// Calls f(integral_constant<IDX>) for the run-time idx in [LO, HI) through a balanced tree of compares (measured 4 %
// faster on a four-instruction program than a switch over the same cases).
template <unsigned LO, unsigned HI, typename F>
__device__ __forceinline__ void tree_dispatch(unsigned idx, F&& f) {
  if constexpr (HI - LO == 1) {
    f(std::integral_constant<unsigned, LO>());
  } else {
    constexpr unsigned MID = (LO + HI) / 2;
    if (idx < MID) tree_dispatch<LO, MID>(idx, f);
    else tree_dispatch<MID, HI>(idx, f);
  }
}

// Division of an index below 2^31 by a fixed extent: q = u * mul >> shift (mul = floor(2^shift / d) + 1, exact there).
struct FastDiv {
  unsigned d, mul;
  int shift;
  __device__ __forceinline__ unsigned div(unsigned u) const { return (unsigned)(((unsigned long long)u * mul) >> shift); }
};
inline FastDiv fast_div(unsigned d) {
  int l = 0;
  while ((1ull << l) < d) ++l;
  return {d, (unsigned)((1ull << (31 + l)) / d + 1), 31 + l};
}
struct Extents {
  long long n;          // elements of the destination
  long long full_below; // a trip that starts at a group below this has all its groups
  FastDiv row, col;     // row: groups (OP_ROW, OP_GROUP, OP_VECTOR) or elements (OP_ELEM) of the first dimension; col: the second extent
  unsigned d0;          // OP_FIXED: the first extent
  int fixed_vec;        // OP_FIXED: the four elements are one aligned vector
  int dest_vec;         // the destination is aligned for vector stores
};

// A group is four neighbouring elements of the destination, whatever the extents are (the last one may be partial); a
// thread owns G groups per trip, a whole grid apart.  The operands of the NEXT trip are copied global -> shared by
// cp.async (no registers, nothing waits on them) while the instructions run on the current trip's copies, so the latency
// of HBM is off the critical path whatever the occupancy; registers hold the accumulator and the current operand,
// and temporaries lie in shared memory too.  A thread reads only the shared memory it filled itself: no CTA barrier anywhere.
// Shared memory: per operand [2 buffers][G][256 threads] groups of 4 * sizeof(T) bytes, OP_FIXED [256 threads]; per temporary [G]
// [256 threads] groups of four floats.
// A trip whose G groups all exist (all but a thread's last) runs without a bounds test.  LINEAR: every operand is laid out
// like the destination, single or fixed (OP_LINEAR, OP_SCALAR, OP_SHIFTED, OP_FIXED), no coordinates are computed.
// What bounds it: HBM for short expressions (A .+ b 6200 GB/s on 8192 x 4096 f32), instruction issue and dispatch latency
// for long ones: a word costs about 24 issue slots of dispatch per thread (16 elements) and half a slot per element for +
// and *.  0.5 v (1 + tanh(c (v + k v^3))), v = A .+ b, on 8192 x 4096 f32: 254 us with a stack of registers, one
// instruction per operator and v evaluated five times; 183 with v in a temporary; 109 with pairs in 64-bit registers
// (107 -> 69 instructions per element); 82 with the words below (7 words, one temporary, b read once); 69.6 with equal
// trips (55 instructions per element, 15 of them moves: a temporary in registers is copied wherever the paths of the words
// meet); 61.1 with the temporary in shared memory, four loads or stores per word that names it. With two temporaries
// (u v + u) / (v v + 1), u = A + b, v = A C: 161 and now 104 us; with three, 207 and 121.
template <typename T, int G, bool TEMPS, bool LINEAR>
__global__ void __launch_bounds__(256, TEMPS ? 3 : 4)
    tiled_broadcast_kernel(void* __restrict__ dest, const Operands in, const Program prog, int n_inputs, const Extents x) {
  ctb::grid_dependency_sync();
  constexpr int V = 4, H = V * G / 2, ES = (int)sizeof(T), VB = V * ES;
  extern __shared__ __align__(16) unsigned char tiled_smem[];
  const long long total = (x.n + V - 1) / V;  // groups
  const long long grid_stride = (long long)gridDim.x * blockDim.x;
  const unsigned tid = threadIdx.x;
  const unsigned smem0 = smem_addr(tiled_smem) + tid * VB;
  auto slot = [&](unsigned buf, unsigned a) { return smem0 + in.slot[a] + buf * (G * 256 * VB); };
  auto element = [&](unsigned buf, unsigned a, int g) {  // of OP_GROUP
    return smem_addr(tiled_smem) + in.slot[a] + ((buf * G + g) * 256 + tid) * ES;
  };

  long long i = (long long)blockIdx.x * blockDim.x + tid;

  auto issue = [&](long long at, unsigned buf, auto full_tag) {
    constexpr bool FULL = decltype(full_tag)::value;
    auto live_of = [&](int g) -> int {  // elements of the trip's group g that exist
      return FULL ? V : (int)max(0ll, min((long long)V, x.n - (at + g * grid_stride) * V));
    };
#pragma unroll
    for (int a = 0; a < kMaxInputs; ++a) {
      if (a >= n_inputs) break;  // uniform, and so are the modes
      const int mode = in.mode[a];
      const T* base = static_cast<const T*>(in.ptr[a]);
      const unsigned to = slot(buf, a);
      if (mode == OP_LINEAR) {
        const char* src = reinterpret_cast<const char*>(base) + at * VB;
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int live = live_of(g);
          cp_async_group<VB>(to + g * (256 * VB), live ? src + g * (grid_stride * VB) : reinterpret_cast<const char*>(base), live * ES);
        }
      } else if (!LINEAR && mode == OP_VECTOR) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int live = live_of(g);
          const unsigned u = live ? (unsigned)at + g * (unsigned)grid_stride : 0u;
          const unsigned i0 = u - x.row.div(u) * x.row.d;
          cp_async_group<VB>(to + g * (256 * VB), base + (unsigned long long)i0 * V, live * ES);
        }
      } else if (mode == OP_SHIFTED) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int live = live_of(g);
          const T* src = base + (at + g * grid_stride) * V;
#pragma unroll
          for (int e = 0; e < V; ++e) copy_element<T>(to + g * (256 * VB) + e * ES, e < live ? src + e : base, e < live);
        }
      } else if (!LINEAR && (mode == OP_ROW || mode == OP_GROUP)) {  // a group exists as a whole or not at all
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int live = live_of(g);
          const unsigned u = live ? (unsigned)at + g * (unsigned)grid_stride : 0u;
          const unsigned r = x.row.div(u), i0 = (u - r * x.row.d) * V, i2 = x.col.div(r), i1 = r - i2 * x.col.d;
          const T* src = base + (i0 * in.stride[a][0] + i1 * in.stride[a][1] + i2 * in.stride[a][2]);
          if (mode == OP_ROW) cp_async_group<VB>(to + g * (256 * VB), src, live * ES);
          else copy_element<T>(element(buf, a, g), src, live != 0);
        }
      } else if (!LINEAR && mode == OP_ELEM) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const int live = live_of(g);
          const unsigned u = live ? ((unsigned)at + g * (unsigned)grid_stride) * V : 0u;
          const unsigned r = x.row.div(u);
          unsigned i0 = u - r * x.row.d, i2 = x.col.div(r), i1 = r - i2 * x.col.d;
#pragma unroll
          for (int e = 0; e < V; ++e) {
            const T* src = base + (i0 * in.stride[a][0] + i1 * in.stride[a][1] + i2 * in.stride[a][2]);
            copy_element<T>(to + g * (256 * VB) + e * ES, e < live ? src : base, e < live);
            if (++i0 == x.row.d) {
              i0 = 0;
              if (++i1 == x.col.d) { i1 = 0; ++i2; }
            }
          }
        }
      }
    }
    cp_async_commit();
  };
  // the elements of every group of operand `a`
  auto fetch = [&](unsigned buf, unsigned arg, Pair (&t)[H]) {
    const unsigned a = arg & (kMaxInputs - 1);
    if (in.mode[a] == OP_SCALAR) {
      const float c = load1<T>(in.ptr[a], 0);
#pragma unroll
      for (int h = 0; h < H; ++h) t[h] = pair(c, c);
      return;
    }
    if (in.mode[a] == OP_FIXED) {
      Pair lo, hi;
      if constexpr (sizeof(T) == 4) {
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "r"(smem0 + in.slot[a]));
      } else {
        uint2 q;
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(q.x), "=r"(q.y) : "r"(smem0 + in.slot[a]));
        const float2 l = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
        lo = pair(l.x, l.y);
        hi = pair(h.x, h.y);
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        t[2 * g] = lo;
        t[2 * g + 1] = hi;
      }
      return;
    }
    if (!LINEAR && in.mode[a] == OP_GROUP) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float c;
        if constexpr (sizeof(T) == 4) {
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(c) : "r"(element(buf, a, g)));
        } else {
          unsigned short h;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(element(buf, a, g)));
          c = __half2float(__ushort_as_half(h));
        }
        t[2 * g] = t[2 * g + 1] = pair(c, c);
      }
      return;
    }
    const unsigned base = slot(buf, a);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if constexpr (sizeof(T) == 4) {
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(t[2 * g]), "=l"(t[2 * g + 1]) : "r"(base + g * (256 * VB)));
      } else {
        uint2 q;
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(q.x), "=r"(q.y) : "r"(base + g * (256 * VB)));
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
        const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
        t[2 * g] = pair(lo.x, lo.y);
        t[2 * g + 1] = pair(hi.x, hi.y);
      }
    }
  };
  const unsigned temps = smem_addr(tiled_smem) + prog.temp_slot + tid * 16;  // [temporary][G][256 threads] groups of four floats
  auto load_temp = [&](unsigned k, Pair (&t)[H]) {
#pragma unroll
    for (int g = 0; g < G; ++g)
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(t[2 * g]), "=l"(t[2 * g + 1]) : "r"(temps + (k * G + g) * 4096) : "memory");
  };
  auto start_next = [&](long long at, unsigned buf) {
    if (at < x.full_below) issue(at, buf, std::true_type());
    else if (at < total) issue(at, buf, std::false_type());
    else cp_async_commit();  // an empty group keeps the count in the wait below uniform
  };

  for (int a = 0; a < n_inputs; ++a) {
    if (in.mode[a] == OP_FIXED) {
      const T* base = static_cast<const T*>(in.ptr[a]);
      const unsigned to = smem0 + in.slot[a];
      unsigned i0 = ((unsigned)i * V) % x.d0;  // the grid is small: 32 bits
      if (x.fixed_vec) {
        cp_async_group<VB>(to, base + i0, VB);
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e) {
          copy_element<T>(to + e * ES, base + i0, true);
          if (++i0 == x.d0) i0 = 0;
        }
      }
    }
  }
  start_next(i, 0);
  for (unsigned buf = 0; i < total; i += grid_stride * G, buf ^= 1u) {
    start_next(i + grid_stride * G, buf ^ 1u);
    cp_async_wait<1>();  // everything but the newest group has landed: this trip's operands

    Pair s0[H];  // the accumulator (every program starts with a load)
    unsigned next = prog.ins[0];  // the word of the next instruction is fetched while the current one runs
    for (int k = 0; k < prog.n_ins; ++k) {
      const unsigned w = next, arg = (w >> 8) & 3u, idx = w & 0xffu;
      const float p = prog.pq[k].x, q = prog.pq[k].y;
      next = prog.ins[k + 1];  // one word of padding behind the last
      if (idx < L_HOT) {
        tree_dispatch<0, 8>(idx, [&](auto tag) {
          constexpr unsigned IDX = decltype(tag)::value;
          if constexpr (IDX == L_FMA) {
            const Pair pp = pair(p, p), qq = pair(q, q);
#pragma unroll
            for (int h = 0; h < H; ++h) s0[h] = fma_pair(s0[h], pp, qq);
          } else if constexpr (IDX == L_LOAD_INPUT) {
            fetch(buf, arg, s0);
          } else if constexpr (IDX == L_LOAD_CONST) {
#pragma unroll
            for (int h = 0; h < H; ++h) s0[h] = pair(q, q);
          } else {
            const float sign = w & kSubtract ? -1.f : 1.f;
            auto apply = [&](Pair (&t)[H]) {
#pragma unroll
              for (int h = 0; h < H; ++h) {
                if constexpr (IDX == L_MUL_INPUT || IDX == L_MUL_TEMP) s0[h] = mul_pair(s0[h], t[h]);
                else s0[h] = fma_pair(t[h], pair(sign, sign), s0[h]);
              }
            };
            if constexpr (IDX == L_LOAD_TEMP) {
              if constexpr (TEMPS) load_temp(arg, s0);
            } else {
              Pair t[H];
              if constexpr (IDX == L_MUL_INPUT || IDX == L_ADD_INPUT) fetch(buf, arg, t);
              else if constexpr (TEMPS) load_temp(arg, t);
              if (TEMPS && (w & kOperandFma)) {
                const Pair pp = pair(p, p), qq = pair(q, q);
#pragma unroll
                for (int h = 0; h < H; ++h) t[h] = fma_pair(t[h], pp, qq);
              }
              if constexpr (TEMPS || IDX == L_MUL_INPUT || IDX == L_ADD_INPUT) apply(t);
            }
          }
        });
      } else {
        tree_dispatch<L_UNARY, L_COUNT>(idx, [&](auto tag) {
          constexpr unsigned IDX = decltype(tag)::value;
          if constexpr (IDX < L_BINARY) {
            apply_unary<(int)(CTB_TILED_NEG + IDX - L_UNARY)>(s0);
          } else {
            constexpr unsigned SRC = (IDX - L_BINARY) / 10, POS = (IDX - L_BINARY) % 10;
            constexpr int CODE = kColdCodes[POS / 2];
            constexpr bool REV = POS & 1u;
            if constexpr (CODE == CTB_TILED_SUB && (SRC == 1 || !REV)) {
              // an L_FMA or L_ADD instruction
            } else if constexpr (SRC == 0) {
              Pair t[H];
              fetch(buf, arg, t);
              apply_binary<CODE, REV>(s0, [&](int h) { return t[h]; });
            } else if constexpr (SRC == 1) {
              apply_binary<CODE, REV>(s0, [&](int) { return pair(q, q); });
            } else {
              if constexpr (TEMPS) {
                Pair t[H];
                load_temp(arg, t);
                apply_binary<CODE, REV>(s0, [&](int h) { return t[h]; });
              }
            }
          }
        });
      }
      if (w >= kTailFma) {
        if (w & kTailFma) {
          const Pair pp = pair(p, p), qq = pair(q, q);
#pragma unroll
          for (int h = 0; h < H; ++h) s0[h] = fma_pair(s0[h], pp, qq);
        }
        if (TEMPS && w >> kTailStore) {
          const unsigned to = temps + ((w >> kTailStore) - 1u) * (G * 4096);
#pragma unroll
          for (int g = 0; g < G; ++g)
            asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(to + g * 4096), "l"(s0[2 * g]), "l"(s0[2 * g + 1]) : "memory");
        }
      }
    }
    if (i < x.full_below && x.dest_vec) {
      char* out = static_cast<char*>(dest) + i * VB;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if constexpr (sizeof(T) == 4) {
          asm volatile("st.global.cs.v2.b64 [%0], {%1, %2};" ::"l"(out + g * (grid_stride * VB)), "l"(s0[2 * g]), "l"(s0[2 * g + 1])
                       : "memory");
        } else {
          const float2 a = unpair(s0[2 * g]), b = unpair(s0[2 * g + 1]);
          uint2 h;
          *reinterpret_cast<__half2*>(&h.x) = __floats2half2_rn(a.x, a.y);
          *reinterpret_cast<__half2*>(&h.y) = __floats2half2_rn(b.x, b.y);
          __stcs(reinterpret_cast<uint2*>(out + g * (grid_stride * VB)), h);
        }
      }
    } else {  // a partial group, or a destination without vector stores
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const long long at = (i + g * grid_stride) * V;
        const float2 a = unpair(s0[2 * g]), b = unpair(s0[2 * g + 1]);
        const float r[V] = {a.x, a.y, b.x, b.y};
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (at + e < x.n) store1<T>(dest, at + e, r[e]);
      }
    }
  }
  cp_async_wait<0>();
}

// CTAs of a broadcast with `groups` groups of four elements per thread and trip.
struct Grid {
  long long ctas, fixed;  // fixed: with operands that vary along the first dimension only; 0: they are read with every group
};
Grid broadcast_grid(ctb_ctx* ctx, long long n, long long d0, int groups) {
  // Several waves of CTAs, not one wave of resident ones: CTAs that all start together stay in step (all loading,
  // then all storing) and measured 10 % slower than CTAs that start at different times.  At most 16 per SM, and as many
  // as give every CTA the same number of trips (2368 CTAs with three or four trips each: 81.8 us for a bias and tanh
  // expression on 8192 x 4096, 2048 with four: 68.5).
  const long long ctas = std::max<long long>(1, ((n + 3) / 4 + 256ll * groups - 1) / (256ll * groups));
  const long long most = (long long)ctx->sm_count * 16, trips = (ctas + most - 1) / most;
  const long long grid = (ctas + trips - 1) / trips;
  // An operand that varies along the first dimension only is the same for all groups of a thread when a whole grid is a
  // multiple of the first extent: a grid of a multiple of m CTAs.  Its four elements are then read once instead of with
  // every group (8192 x 4096, A .+ b: 20.8 -> 14 instructions per element).
  const long long m = d0 / std::min(d0 & -d0, 1024ll);  // over the common divisor with 256 threads of four elements
  const long long up = (grid + m - 1) / m * m;
  return {grid, up <= std::max(most, std::min(ctas, 4 * most)) ? up : grid / m * m};
}
bool along_first(const Operands& in, int a) {
  return in.mode[a] == OP_VECTOR || (in.mode[a] == OP_ELEM && in.stride[a][0] == 1 && !in.stride[a][1] && !in.stride[a][2]);
}
// Bytes of shared memory of an operand with elements of `es` bytes.
size_t operand_bytes(int mode, int groups, int es) {
  return mode == OP_SCALAR ? 0 : (size_t)256 * es * (mode == OP_FIXED ? 4 : mode == OP_GROUP ? 2 * groups : 8 * groups);
}

template <typename T, int G, bool TEMPS>
int launch_broadcast(ctb_ctx* ctx, cudaStream_t st, void* dest, Operands& in, Program& prog, int n_inputs, long long d0,
                     Extents& x) {
  constexpr int VB = 4 * (int)sizeof(T);
  const Grid grids = broadcast_grid(ctx, x.n, d0, G);
  long long grid = grids.ctas;
  bool linear = true, fixed = false;
  for (int a = 0; a < n_inputs; ++a) {
    if (along_first(in, a) && grids.fixed > 0) {
      in.mode[a] = OP_FIXED;
      fixed = true;
    } else if (in.mode[a] == OP_VECTOR || in.mode[a] == OP_ROW || in.mode[a] == OP_GROUP || in.mode[a] == OP_ELEM) {
      linear = false;
    }
  }
  if (fixed) {
    grid = grids.fixed;
    x.d0 = (unsigned)d0;
    x.fixed_vec = d0 % 4 == 0;
    for (int a = 0; a < n_inputs; ++a)
      if (in.mode[a] == OP_FIXED && (uintptr_t)in.ptr[a] % VB) x.fixed_vec = 0;
  }
  unsigned smem = 0;
  for (int a = 0; a < n_inputs; ++a) {
    in.slot[a] = smem;
    smem += (unsigned)operand_bytes(in.mode[a], G, sizeof(T));
  }
  prog.temp_slot = smem;
  smem += prog.n_temps * G * 4096;
  x.full_below = x.n / 4 - (long long)(G - 1) * grid * 256;  // a trip's last group is (G - 1) grids further on
  auto kernel = linear ? tiled_broadcast_kernel<T, G, TEMPS, true> : tiled_broadcast_kernel<T, G, TEMPS, false>;
  if (smem > 48 * 1024 &&  // per device, so on every launch that needs it: a host-side table write
      allow_smem(kernel, (size_t)kMaxInputs * 2 * G * 256 * VB + (TEMPS ? kTemps * G * 4096 : 0)) != cudaSuccess)
    return fail(CTB_CUDA_ERROR, "ctb_tiled_broadcast: shared memory attribute: %s", cudaGetErrorString(cudaGetLastError()));
  launch_kernel(kernel, (unsigned)grid, 256, smem, st, 0, dest, in, prog, n_inputs, x);
  return CTB_OK;
}

// ---- mapreduce ----------------------------------------------------------------------------------------------------
__device__ __forceinline__ float neutral(int op) {
  return op == CTB_TILED_ADD ? 0.f : op == CTB_TILED_MUL ? 1.f : op == CTB_TILED_MAX ? -INFINITY : INFINITY;
}

struct ReduceShape {
  long long d[3];        // extents
  long long keep_n[3];   // extent of each dimension in the output index space (1 when reduced)
  long long red_n[3];    // extent of each dimension in the reduced index space (1 when kept)
  long long outputs, red_len, parts, chunk;
};

// A reduction that is cut into parts leaves one partial result per (part, output) in the stream's scratch, outputs
// contiguous; the CTA that finishes last for its outputs (a counter per grid column, which its arrival returns to zero) adds
// the parts up in a fixed order.  One launch instead of two, and the result does not depend on which CTA is last.
// True for every thread of the last CTA; the partials of the others are visible then.
__device__ __forceinline__ bool last_part(unsigned* ticket, long long parts) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {  // its fences cover what the barrier has ordered before and behind them
    __threadfence();
    last = atomicInc(ticket, (unsigned)parts - 1) == (unsigned)parts - 1;
    __threadfence();
  }
  __syncthreads();
  return last != 0;
}

// The first dimension is reduced: one CTA per (output, part).  The reduced index space is the first
// dimension (contiguous) times the other reduced dimensions ("rows"); a part is a range [lo, hi) of it.  The CTA walks
// its rows one after the other, inside a row 16 bytes per thread and trip where the row starts on a 16-byte boundary,
// and combines in a fixed order (thread partials, lanes, then warps in order).
// OP is a compile-time constant and so is "f is the identity": a dispatch per element would cost more than the element.
template <typename T, int OP, bool MAPPED>
__global__ void __launch_bounds__(256)
    tiled_reduce_rows_kernel(const void* __restrict__ src, float* __restrict__ partial, void* __restrict__ dest,
                             const ReduceShape s, int f_code, unsigned* tickets) {
  ctb::grid_dependency_sync();
  constexpr int op = OP;
  auto fmap = [&](float v) { return MAPPED ? unary(f_code, v) : v; };
  __shared__ float wsum[8];
  auto block_combine = [&](float acc) {  // valid in thread 0; the CTA has met since an earlier call
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) acc = binary(op, acc, __shfl_xor_sync(0xffffffffu, acc, sh));
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      acc = wsum[0];
      for (int w = 1; w < 8; ++w) acc = binary(op, acc, wsum[w]);
    }
    return acc;
  };
  const long long part = blockIdx.y;
  const long long lo = part * s.chunk, hi = min(s.red_len, lo + s.chunk);
  const long long st1 = s.d[0], st2 = s.d[0] * s.d[1];  // element strides of dimensions 1 and 2
  // output coordinates: the first dimension is reduced, so the output index runs over dimensions 1 and 2
  const long long o = blockIdx.x;
  const long long k1 = o % s.keep_n[1], k2 = o / s.keep_n[1];
  const long long base = k1 * st1 + k2 * st2;
  const long long d0 = s.d[0];
  constexpr int V = 16 / sizeof(T);
  float acc = neutral(op);
  long long row = lo / d0, r1 = row % s.red_n[1], r2 = row / s.red_n[1];
  for (; row * d0 < hi; ++row, ++r1) {  // rows of the reduced index space that this part touches
    if (r1 == s.red_n[1]) {
      r1 = 0;
      ++r2;
    }
    const long long rbase = base + r1 * st1 + r2 * st2;
    const long long c_lo = max(lo - row * d0, 0ll), c_hi = min(hi - row * d0, d0);
    const bool vec = ((rbase + c_lo) * (long long)sizeof(T) + (long long)(uintptr_t)src) % 16 == 0;
    const long long c_vec = vec ? c_lo + (c_hi - c_lo) / V * V : c_lo;
    for (long long c = c_lo + (long long)threadIdx.x * V; c < c_vec; c += 256 * V) {
      if constexpr (sizeof(T) == 4) {
        const float4 q = __ldcs(reinterpret_cast<const float4*>(static_cast<const float*>(src) + rbase + c));
        acc = binary(op, acc, fmap(q.x));
        acc = binary(op, acc, fmap(q.y));
        acc = binary(op, acc, fmap(q.z));
        acc = binary(op, acc, fmap(q.w));
      } else {
        const uint4 q = __ldcs(reinterpret_cast<const uint4*>(static_cast<const __half*>(src) + rbase + c));
        const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 v = __half22float2(h[j]);
          acc = binary(op, acc, fmap(v.x));
          acc = binary(op, acc, fmap(v.y));
        }
      }
    }
    for (long long c = c_vec + threadIdx.x; c < c_hi; c += 256) acc = binary(op, acc, fmap(load1<T>(src, rbase + c)));
  }
  acc = block_combine(acc);
  if (s.parts == 1) {
    if (threadIdx.x == 0) store1<T>(dest, o, acc);
    return;
  }
  if (threadIdx.x == 0) partial[part * s.outputs + o] = acc;
  if (!last_part(tickets + o, s.parts)) return;
  acc = neutral(op);
  for (long long q = threadIdx.x; q < s.parts; q += 256) acc = binary(op, acc, __ldcg(partial + q * s.outputs + o));
  acc = block_combine(acc);
  if (threadIdx.x == 0) store1<T>(dest, o, acc);
}

// The first dimension is kept.  A thread owns VB neighbouring outputs (one 16-byte load fetches an element of each when
// the first extent and the source allow it, VB = 1 otherwise); 2^lx such groups side by side and 256 / 2^lx slices of the
// reduced index space make a CTA, whose slices meet in shared memory in ascending order.  Whatever dimensions are
// reduced, consecutive elements of the reduced index space are `rstride` apart.  Eight loads in flight per thread.
// Bound by HBM.  With a thread per output over one long slice, the parts (293 for 8192 x 4096) were written 4 bytes at a
// time a part count apart and added up by one thread per output: 31 + 35 us for the 134 MB; with the slices of a CTA
// combined on chip (18 parts, 512 contiguous bytes per warp and row, the last CTA adds the parts): 25 us.
template <typename T, int OP, bool MAPPED, int VB>
__global__ void __launch_bounds__(256)
    tiled_reduce_cols_kernel(const void* __restrict__ src, float* __restrict__ partial, void* __restrict__ dest,
                             const ReduceShape s, long long rstride, int lx, int f_code, unsigned* tickets) {
  ctb::grid_dependency_sync();
  constexpr int op = OP;
  auto fmap = [&](float v) { return MAPPED ? unary(f_code, v) : v; };
  __shared__ float meet[256][VB];
  const int LX = 1 << lx, slices = 256 >> lx;
  const int cx = threadIdx.x & (LX - 1), slice = threadIdx.x >> lx;
  const long long groups = s.outputs / VB, group = (long long)blockIdx.x * LX + cx, o = group * VB;
  const long long part = blockIdx.y, p_lo = part * s.chunk, p_hi = min(s.red_len, p_lo + s.chunk);
  const long long per = (p_hi - p_lo + slices - 1) / slices;
  const long long lo = min(p_hi, p_lo + slice * per), hi = min(p_hi, lo + per);
  // VB elements as they lie in memory, so that eight loads in flight cost eight vectors of registers
  using Raw = std::conditional_t<VB == 1, T, std::conditional_t<VB * sizeof(T) == 16, uint4, uint2>>;
  auto value = [](const Raw& x, int e) -> float {
    if constexpr (VB == 1) {
      if constexpr (sizeof(T) == 4) return x;
      else return __half2float(x);
    } else if constexpr (sizeof(T) == 4) {
      return reinterpret_cast<const float*>(&x)[e];
    } else {
      return __half2float(reinterpret_cast<const __half*>(&x)[e]);
    }
  };
  float acc[VB];
#pragma unroll
  for (int e = 0; e < VB; ++e) acc[e] = neutral(op);
  if (group < groups) {
    const long long k0 = o % s.keep_n[0], q = o / s.keep_n[0], k1 = q % s.keep_n[1], k2 = q / s.keep_n[1];
    const long long base = k0 + k1 * s.d[0] + k2 * s.d[0] * s.d[1];
    const char* at = static_cast<const char*>(src) + (base + lo * rstride) * (long long)sizeof(T);
    const long long step = rstride * (long long)sizeof(T);
    constexpr int kFlight = VB == 1 ? 16 : 8;
    for (long long r = lo; r < hi; r += kFlight) {
      Raw v[kFlight];
#pragma unroll
      for (int j = 0; j < kFlight; ++j)
        if (r + j < hi) v[j] = __ldcs(reinterpret_cast<const Raw*>(at + j * step));
      at += kFlight * step;
#pragma unroll
      for (int j = 0; j < kFlight; ++j)
        if (r + j < hi)
#pragma unroll
          for (int e = 0; e < VB; ++e) acc[e] = binary(op, acc[e], fmap(value(v[j], e)));
    }
  }
  // slices in ascending order
  if (slices > 1) {
#pragma unroll
    for (int e = 0; e < VB; ++e) meet[threadIdx.x][e] = acc[e];
    __syncthreads();
    if (slice == 0) {
      for (int k = 1; k < slices; ++k)
#pragma unroll
        for (int e = 0; e < VB; ++e) acc[e] = binary(op, acc[e], meet[(k << lx) + cx][e]);
    }
  }
  auto finish = [&]() {
    if (slice == 0 && group < groups)
#pragma unroll
      for (int e = 0; e < VB; ++e) store1<T>(dest, o + e, acc[e]);
  };
  if (s.parts == 1) {
    finish();
    return;
  }
  if (slice == 0 && group < groups)
#pragma unroll
    for (int e = 0; e < VB; ++e) partial[part * s.outputs + o + e] = acc[e];
  if (!last_part(tickets + blockIdx.x, s.parts)) return;
  // the parts: slice k takes parts k, k + slices, ... (their loads overlap), then the slices meet as above
#pragma unroll
  for (int e = 0; e < VB; ++e) acc[e] = neutral(op);
  if (group < groups) {
    constexpr int kParts = 8;
    for (long long q0 = slice; q0 < s.parts; q0 += (long long)kParts * slices) {
      float v[kParts][VB];
#pragma unroll
      for (int j = 0; j < kParts; ++j) {
        const long long q = q0 + (long long)j * slices;
#pragma unroll
        for (int e = 0; e < VB; ++e) v[j][e] = neutral(op);
        if (q < s.parts) {
          const float* src_p = partial + q * s.outputs + o;
          if constexpr (VB % 4 == 0) {
#pragma unroll
            for (int e = 0; e < VB; e += 4) {
              const float4 x = __ldcg(reinterpret_cast<const float4*>(src_p + e));
              v[j][e] = x.x; v[j][e + 1] = x.y; v[j][e + 2] = x.z; v[j][e + 3] = x.w;
            }
          } else {
            v[j][0] = __ldcg(src_p);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kParts; ++j)
#pragma unroll
        for (int e = 0; e < VB; ++e) acc[e] = binary(op, acc[e], v[j][e]);
    }
  }
  if (slices > 1) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < VB; ++e) meet[threadIdx.x][e] = acc[e];
    __syncthreads();
    if (slice == 0) {
      for (int k = 1; k < slices; ++k)
#pragma unroll
        for (int e = 0; e < VB; ++e) acc[e] = binary(op, acc[e], meet[(k << lx) + cx][e]);
    }
  }
  finish();
}

}  // namespace

extern "C" {

int ctb_tiled_broadcast(ctb_ctx* ctx, void* stream, void* dest, const int64_t* shape, const void* const* inputs,
                        const int64_t* input_strides, int n_inputs, const int32_t* program, int n_ops, const float* constants,
                        int n_constants, int dtype) {
  CTB_CHECK_CTX(ctx);
  if (!shape || !program) return fail(CTB_BAD_ARG, "ctb_tiled_broadcast: null shape or program");
  if (dtype != CTB_F32 && dtype != CTB_F16) return fail(CTB_UNSUPPORTED, "ctb_tiled_broadcast: element type must be f32 or f16");
  if (n_inputs < 0 || n_inputs > kMaxInputs || n_ops < 1 || n_ops > kMaxOps || n_constants < 0 || n_constants > kMaxConsts)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_broadcast: at most %d inputs, %d operations and %d constants", kMaxInputs, kMaxOps,
                kMaxConsts);
  if ((n_inputs && (!inputs || !input_strides)) || (n_constants && !constants))
    return fail(CTB_BAD_ARG, "ctb_tiled_broadcast: null operand table");
  for (int k = 0; k < 3; ++k)
    if (shape[k] < 0) return fail(CTB_BAD_ARG, "ctb_tiled_broadcast: negative extent");
  Program prog;
  const char* why = "";
  const int bad = lower_program(program, n_ops, n_inputs, constants, n_constants, &prog, &why);
  if (bad == -1000)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_broadcast: the expression needs more than %d intermediate values at once", kStack);
  if (bad) return fail(CTB_BAD_ARG, "ctb_tiled_broadcast: operation %d %s", -bad - 1, why);
  const long long d0 = shape[0], d1 = shape[1], d2 = shape[2];
  if (d0 == 0 || d1 == 0 || d2 == 0) return CTB_OK;  // empty arrays: nothing to launch
  CTB_CHECK_DEV(dest);
  const int es = dtype == CTB_F32 ? 4 : 2;
  Operands in = {};
  Extents x = {};
  x.n = d0 * d1 * d2;
  x.dest_vec = (uintptr_t)dest % (4 * es) == 0;
  bool linear = true, by_element = false;
  for (int a = 0; a < n_inputs; ++a) {
    CTB_CHECK_DEV(inputs[a]);
    in.ptr[a] = inputs[a];
    for (int k = 0; k < 3; ++k) {
      in.stride[a][k] = input_strides[3 * a + k];
      if (in.stride[a][k] < 0) return fail(CTB_BAD_ARG, "ctb_tiled_broadcast: negative stride");
    }
    const long long s0 = in.stride[a][0], s1 = in.stride[a][1], s2 = in.stride[a][2];
    const bool like_dest = (d0 == 1 || s0 == 1) && (d1 == 1 || s1 == d0) && (d2 == 1 || s2 == d0 * d1);
    const bool single = (d0 == 1 || s0 == 0) && (d1 == 1 || s1 == 0) && (d2 == 1 || s2 == 0);
    const bool aligned = (uintptr_t)inputs[a] % (4 * es) == 0;
    if (single) in.mode[a] = OP_SCALAR;
    else if (like_dest) in.mode[a] = aligned ? OP_LINEAR : OP_SHIFTED;
    else if (d0 % 4 == 0 && s0 == 1 && aligned && s1 == 0 && s2 == 0) in.mode[a] = OP_VECTOR;
    else if (d0 % 4 == 0 && s0 == 0) in.mode[a] = OP_GROUP;
    else if (d0 % 4 == 0 && s0 == 1 && aligned && s1 % 4 == 0 && s2 % 4 == 0) in.mode[a] = OP_ROW;
    else in.mode[a] = OP_ELEM;
    if (in.mode[a] == OP_ROW || in.mode[a] == OP_GROUP || in.mode[a] == OP_ELEM || in.mode[a] == OP_VECTOR) linear = false;
    if (in.mode[a] == OP_ELEM) by_element = true;
  }
  if (by_element)  // one pair of divisors serves both kinds: by element then
    for (int a = 0; a < n_inputs; ++a)
      if (in.mode[a] == OP_ROW || in.mode[a] == OP_GROUP || in.mode[a] == OP_VECTOR) in.mode[a] = OP_ELEM;
  if (!linear) {
    if ((by_element ? x.n : x.n / 4) > 0x7fffffffLL)
      return fail(CTB_UNSUPPORTED, "ctb_tiled_broadcast: too many elements for an expanded operand");
    x.row = fast_div((unsigned)(by_element ? d0 : d0 / 4));
    x.col = fast_div((unsigned)d1);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = CTB_OK;
  // Groups per thread.  With temporaries the most of four, three and two with which three CTAs fit the shared memory of an SM
  // (operands twice, those that stay the same and temporaries once): 8192 x 4096 f32, bias and tanh of A + B, 76.7 us with two, 71.2
  // with three, 76.9 with four; a bias instead of B stays the same, and four fit (60.7, 74.7 with two).  Without temporaries four for
  // up to three operands, although three arrays of f32 leave room for two CTAs only.
  const bool temps = prog.n_temps || prog.operand_fma;
  bool stays = false;  // some operand may stay the same
  for (int a = 0; a < n_inputs; ++a) stays = stays || along_first(in, a);
  auto need = [&](int groups) {
    const bool fixed = stays && broadcast_grid(ctx, x.n, d0, groups).fixed > 0;
    size_t bytes = (size_t)prog.n_temps * groups * 4096;
    for (int a = 0; a < n_inputs; ++a) bytes += operand_bytes(fixed && along_first(in, a) ? OP_FIXED : in.mode[a], groups, es);
    return bytes;
  };
  int groups = n_inputs <= 3 ? 4 : 2;
  if (temps) {
    groups = need(4) <= 72 * 1024 ? 4 : need(3) <= 72 * 1024 ? 3 : 2;
    // Four also where two CTAs per SM are all there are: every CTA reads the operand that stays (f32 tanh of a square of A B + bias,
    // 2450 x 356 5.9 us, 7.2 with three, 8.5 with two; 11064 x 72 7.4, 8.7, 11.2).
    if (stays && groups < 4 && need(4) <= 112 * 1024) {
      const Grid four = broadcast_grid(ctx, x.n, d0, 4);
      if (four.fixed > 0 && four.fixed <= 2 * ctx->sm_count && four.fixed < 2 * four.ctas) groups = 4;
    }
  }
  const Grid grid = broadcast_grid(ctx, x.n, d0, groups);
  if (stays && grid.fixed > 0) {
    // Such a grid may be far larger than the elements need, and a thread then has one group and computes more: two where four groups
    // have twice the CTAs (bias and tanh of 1000 x 1001 in f32 7.5 us, with four 11.4; of 452 x 1988 in f16 4.2 and 7.5), or three a fifth more
    // (4000 x 2001: 2001 CTAs of three groups have 1.3 trips, 31.5 us; of two 1.95, 24.8; but 3459 x 356, 445 CTAs for 401, 7.5 and 8.8).
    // Otherwise four also with few elements (bias and tanh of 11064 x 72 7.0 us, 11.0 with two; the bias alone 5.1 and 10.1).
    if (groups == 3 ? grid.fixed * 10 > grid.ctas * 12 : grid.fixed >= grid.ctas * 2) groups = 2;
  } else if (2 * grid.ctas < (groups == 3 ? 5ll : 4ll) * ctx->sm_count) {
    // Two as well where more would leave fewer than two CTAs per SM, or two and a half with three groups (f32 1000 x 1001: tanh
    // of 2 A + 1 2.8 us, with four 3.6; A + B 2.6 and 3.1).
    groups = 2;
  }
  auto launch = [&](auto zero) {
    using T = decltype(zero);
    if (temps)
      return groups == 4   ? launch_broadcast<T, 4, true>(ctx, st, dest, in, prog, n_inputs, d0, x)
             : groups == 3 ? launch_broadcast<T, 3, true>(ctx, st, dest, in, prog, n_inputs, d0, x)
                           : launch_broadcast<T, 2, true>(ctx, st, dest, in, prog, n_inputs, d0, x);
    return groups == 4 ? launch_broadcast<T, 4, false>(ctx, st, dest, in, prog, n_inputs, d0, x)
                       : launch_broadcast<T, 2, false>(ctx, st, dest, in, prog, n_inputs, d0, x);
  };
  rc = dtype == CTB_F32 ? launch(0.f) : launch(__half());
  if (rc) return rc;
  CTB_CHECK_LAUNCH("ctb_tiled_broadcast launch");
  return CTB_OK;
}

int ctb_tiled_compile(const int32_t* program, int n_ops, int n_inputs, int n_constants, uint32_t* instructions,
                      int* n_instructions) {
  if (!program || !instructions || !n_instructions) return fail(CTB_BAD_ARG, "ctb_tiled_compile: null argument");
  if (n_inputs < 0 || n_inputs > kMaxInputs || n_ops < 1 || n_ops > kMaxOps || n_constants < 0 || n_constants > kMaxConsts)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_compile: at most %d inputs, %d operations and %d constants", kMaxInputs, kMaxOps,
                kMaxConsts);
  Compiler c;
  const char* why = "";
  const int bad = compile_program(program, n_ops, n_inputs, n_constants, &c, &why);
  if (bad == -1000)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_compile: the expression needs more than %d intermediate values at once", kStack);
  if (bad) return fail(CTB_BAD_ARG, "ctb_tiled_compile: operation %d %s", -bad - 1, why);
  for (int k = 0; k < c.n_words; ++k) instructions[k] = c.words[k];
  *n_instructions = c.n_words;
  return CTB_OK;
}

int ctb_tiled_lower(const int32_t* program, int n_ops, int n_inputs, const float* constants, int n_constants, uint32_t* words,
                    float* constants_pq, int* n_words, int* n_temps) {
  if (!program || !words || !constants_pq || !n_words || !n_temps || (n_constants && !constants))
    return fail(CTB_BAD_ARG, "ctb_tiled_lower: null argument");
  if (n_inputs < 0 || n_inputs > kMaxInputs || n_ops < 1 || n_ops > kMaxOps || n_constants < 0 || n_constants > kMaxConsts)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_lower: at most %d inputs, %d operations and %d constants", kMaxInputs, kMaxOps,
                kMaxConsts);
  Program prog;
  const char* why = "";
  const int bad = lower_program(program, n_ops, n_inputs, constants, n_constants, &prog, &why);
  if (bad == -1000)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_lower: the expression needs more than %d intermediate values at once", kStack);
  if (bad) return fail(CTB_BAD_ARG, "ctb_tiled_lower: operation %d %s", -bad - 1, why);
  for (int k = 0; k < prog.n_ins; ++k) {
    words[k] = prog.ins[k];
    constants_pq[2 * k] = prog.pq[k].x;
    constants_pq[2 * k + 1] = prog.pq[k].y;
  }
  *n_words = prog.n_ins;
  *n_temps = prog.n_temps;
  return CTB_OK;
}

int ctb_tiled_mapreduce(ctb_ctx* ctx, void* stream, void* dest, const void* src, const int64_t* shape, int reduce_mask, int f,
                        int op, int dtype) {
  CTB_CHECK_CTX(ctx);
  if (!shape) return fail(CTB_BAD_ARG, "ctb_tiled_mapreduce: null shape");
  if (dtype != CTB_F32 && dtype != CTB_F16) return fail(CTB_UNSUPPORTED, "ctb_tiled_mapreduce: element type must be f32 or f16");
  if (f < CTB_TILED_IDENTITY || f > CTB_TILED_ABS2) return fail(CTB_BAD_ARG, "ctb_tiled_mapreduce: f must be a unary function code");
  if (op != CTB_TILED_ADD && op != CTB_TILED_MUL && op != CTB_TILED_MAX && op != CTB_TILED_MIN)
    return fail(CTB_UNSUPPORTED, "ctb_tiled_mapreduce: the reduction must be +, *, max or min");
  if (reduce_mask < 0 || reduce_mask > 7) return fail(CTB_BAD_ARG, "ctb_tiled_mapreduce: reduce_mask has bits for three dimensions");
  ReduceShape s;
  s.outputs = 1;
  s.red_len = 1;
  for (int k = 0; k < 3; ++k) {
    if (shape[k] < 0) return fail(CTB_BAD_ARG, "ctb_tiled_mapreduce: negative extent");
    s.d[k] = shape[k];
  }
  // Reduced dimensions behind a reduced first one are contiguous with it: one long row instead of many that may be short.
  for (int k = 0; k < 2 && (reduce_mask & 1); ++k)
    if ((reduce_mask & 2) || s.d[1] == 1) {
      s.d[0] *= s.d[1];
      s.d[1] = s.d[2];
      s.d[2] = 1;
      reduce_mask = 1 | ((reduce_mask >> 1) & 2);
    }
  for (int k = 0; k < 3; ++k) {
    const bool red = (reduce_mask >> k) & 1;
    s.keep_n[k] = red ? 1 : s.d[k];
    s.red_n[k] = red ? s.d[k] : 1;
    s.outputs *= s.keep_n[k];
    s.red_len *= s.red_n[k];
  }
  if (s.outputs == 0) return CTB_OK;  // no output elements
  CTB_CHECK_DEV(dest);
  if (s.red_len > 0) CTB_CHECK_DEV(src);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool mode_a = (reduce_mask & 1) != 0 && s.red_len > 0;
  const int es = dtype == CTB_F32 ? 4 : 2;
  const bool mapped = f != CTB_TILED_IDENTITY;
  // the first dimension kept: four neighbouring outputs per thread where the first extent and the source's alignment allow
  // it (f16 with eight, 16-byte loads: 20 us against 17 for 8192 x 4096)
  const int vb = (reduce_mask & 1) == 0 && s.d[0] % 4 == 0 && (uintptr_t)src % (4 * es) == 0 ? 4 : 1;
  const long long groups = s.outputs / vb;
  // the CTA's 256 threads: as many slices of the reduced index space (eight at most) as leave each at least eight
  // elements, more when there are too few outputs to fill the rest
  int lx = 8;
  while (lx > 5 && s.red_len >> (8 - lx) >= 16) --lx;
  while (lx > 0 && (1ll << (lx - 1)) >= groups) --lx;
  const long long columns = mode_a ? s.outputs : (groups + (1ll << lx) - 1) >> lx;  // CTAs side by side
  // parts: eight CTAs per SM in all for the row kernel; for the column kernel one wave of four per SM (its registers allow
  // four; 8192 x 4096 f32: 26 us with 4, 32 with 6, 29 with 8: every further part costs the last CTA's sum).  A part is at
  // least 4096 elements for a row CTA, 16 per slice for a column CTA: two rounds of loads cost less than the last CTA's turn
  // (100 x 8000 f32: 5.0 us with eight, 3.1 with 16; 13885 x 348 f16: 10.1 and 9.2).
  const long long min_part = mode_a ? 4096 : 16ll * (256 >> lx);
  s.parts = std::max<long long>(1, std::min<long long>({(long long)ctx->sm_count * (mode_a ? 8 : 4) / std::max<long long>(1, columns),
                                                        (s.red_len + min_part - 1) / min_part, (long long)1024}));
  if (columns > kTickets) s.parts = 1;  // enough CTAs as it is
  auto cut = [&]() {
    s.chunk = (std::max<long long>(1, s.red_len) + s.parts - 1) / s.parts;
    if (mode_a) s.chunk = (s.chunk + 1023) / 1024 * 1024;  // parts start on 16-byte boundaries of an aligned row
    s.parts = (std::max<long long>(1, s.red_len) + s.chunk - 1) / s.chunk;
  };
  cut();
  // More than one part means at most eight row CTAs with one output or four column CTAs with 128 outputs per SM: 300 KB of
  // partial results on 148 SMs.
  std::optional<StreamScratch> scratch;  // until the kernel is launched
  if (s.parts > 1) {
    scratch.emplace(ctx, st);
    if (!scratch->data || (size_t)(s.outputs * s.parts) * sizeof(float) > kStreamScratchBytes) {
      s.parts = 1;  // one CTA per column takes all of it
      cut();
    }
  }
  float* partial = s.parts > 1 ? scratch->data : nullptr;
  unsigned* tickets = s.parts > 1 ? scratch->tickets : nullptr;
  if (columns > 0x7fffffffLL) return fail(CTB_UNSUPPORTED, "ctb_tiled_mapreduce: too many output elements");
  const dim3 grid((unsigned)columns, (unsigned)s.parts);
  const long long rstride = (reduce_mask & 2) ? s.d[0] : s.d[0] * s.d[1];  // between elements of the reduced index space
#define CTB_RED_LAUNCH(T, OP, M)                                                                                            \
  do {                                                                                                                      \
    if (mode_a)                                                                                                             \
      launch_kernel(tiled_reduce_rows_kernel<T, OP, M>, grid, 256, 0, st, 0, src, partial, dest, s, f, tickets);       \
    else if (vb == 4)                                                                                                       \
      launch_kernel(tiled_reduce_cols_kernel<T, OP, M, 4>, grid, 256, 0, st, 0, src, partial, dest, s, rstride, lx, f,      \
                    tickets);                                                                                          \
    else                                                                                                                    \
      launch_kernel(tiled_reduce_cols_kernel<T, OP, M, 1>, grid, 256, 0, st, 0, src, partial, dest, s, rstride, lx, f,      \
                    tickets);                                                                                          \
  } while (0)
#define CTB_RED_MAPPED(T, OP)              \
  do {                                     \
    if (mapped) CTB_RED_LAUNCH(T, OP, true); \
    else CTB_RED_LAUNCH(T, OP, false);     \
  } while (0)
#define CTB_RED_OP(T)                                              \
  do {                                                             \
    if (op == CTB_TILED_ADD) CTB_RED_MAPPED(T, CTB_TILED_ADD);     \
    else if (op == CTB_TILED_MUL) CTB_RED_MAPPED(T, CTB_TILED_MUL); \
    else if (op == CTB_TILED_MAX) CTB_RED_MAPPED(T, CTB_TILED_MAX); \
    else CTB_RED_MAPPED(T, CTB_TILED_MIN);                         \
  } while (0)
  if (dtype == CTB_F32) CTB_RED_OP(float);
  else CTB_RED_OP(__half);
#undef CTB_RED_OP
#undef CTB_RED_MAPPED
#undef CTB_RED_LAUNCH
  CTB_CHECK_LAUNCH("ctb_tiled_mapreduce launch");
  return CTB_OK;
}

}  // extern "C"
