// pa_cholesky_order_check: the order in which the two streams of the Cholesky
// factorization (k_linalg.cu) run its launches. The factorization of an n x n
// matrix is captured into a graph, which is read and never launched, so the
// order is checked for every n without a race having to show itself.
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "k_linalg.cuh"
#include "pa_b200.h"

namespace pa {
int set_error(int code, const std::string& msg);
}  // namespace pa

namespace {

constexpr int kCols = 64;  // columns of a step

struct Order {
  int missing = 0, apart = 0, pairs = 0;
};

cudaError_t read_order(cudaGraph_t graph, int n, Order* out) {
  size_t nn = 0, ne = 0;
  cudaError_t e = cudaGraphGetNodes(graph, nullptr, &nn);
  if (e == cudaSuccess) e = cudaGraphGetEdges(graph, nullptr, nullptr, &ne);
  std::vector<cudaGraphNode_t> nodes(nn), from(ne), to(ne);
  if (e == cudaSuccess) e = cudaGraphGetNodes(graph, nodes.data(), &nn);
  if (e == cudaSuccess) e = cudaGraphGetEdges(graph, from.data(), to.data(), &ne);
  if (e != cudaSuccess) return e;
  std::map<cudaGraphNode_t, int> id;
  for (size_t i = 0; i < nn; ++i) id[nodes[i]] = static_cast<int>(i);
  std::vector<std::vector<int>> next(nn);
  for (size_t i = 0; i < ne; ++i) next[id[from[i]]].push_back(id[to[i]]);
  std::vector<std::vector<char>> before(nn, std::vector<char>(nn, 0));  // before[a][b]: a runs before b
  for (size_t a = 0; a < nn; ++a) {
    std::vector<int> todo(next[a]);
    while (!todo.empty()) {
      const int b = todo.back();
      todo.pop_back();
      if (before[a][b]) continue;
      before[a][b] = 1;
      todo.insert(todo.end(), next[b].begin(), next[b].end());
    }
  }
  std::map<int, int> step, update;  // block column -> node
  for (size_t i = 0; i < nn; ++i) {
    cudaGraphNodeType type;
    e = cudaGraphNodeGetType(nodes[i], &type);
    if (e != cudaSuccess) return e;
    if (type != cudaGraphNodeTypeKernel) continue;
    cudaKernelNodeParams p{};
    e = cudaGraphKernelNodeGetParams(nodes[i], &p);
    const char* name = nullptr;
    if (e == cudaSuccess) e = cudaFuncGetName(&name, p.func);
    if (e != cudaSuccess) return e;
    if (std::strstr(name, "k_chol_step"))
      step[*static_cast<const int*>(p.kernelParams[3])] = static_cast<int>(i);  // (A, lda, n, c, ..)
    else if (std::strstr(name, "k_syrk_update"))
      update[(n - *static_cast<const int*>(p.kernelParams[0])) / kCols - 2] = static_cast<int>(i);  // m = n - 64 (c + 2)
  }
  // step c takes the contribution of column c - 1 itself, so it needs the
  // updates up to that of column c - 2; the update of column c needs step c and
  // the update before it
  const int nblk = (n + kCols - 1) / kCols;
  auto needs = [&](const std::map<int, int>& a, int ca, const std::map<int, int>& b, int cb) {
    if (a.count(ca) && b.count(cb) && !before[a.at(ca)][b.at(cb)]) ++out->missing;
  };
  for (int c = -1; c + 1 < nblk; ++c) {
    if (!step.count(c)) ++out->missing;
    if (n - (c + 2) * kCols > kCols && c >= 0 && !update.count(c)) ++out->missing;
    needs(step, c - 1, step, c);
    needs(update, c - 2, step, c);
    needs(step, c, update, c);
    needs(update, c - 1, update, c);
    if (update.count(c - 1) && step.count(c)) {
      ++out->pairs;
      if (!before[update.at(c - 1)][step.at(c)] && !before[step.at(c)][update.at(c - 1)]) ++out->apart;
    }
  }
  return cudaSuccess;
}

}  // namespace

extern "C" int pa_cholesky_order_check(int n, int* missing, int* apart, int* pairs) {
  if (n < 1 || n > 16384 || !missing || !apart || !pairs)
    return pa::set_error(PA_ERR_ARG, "pa_cholesky_order_check: need 1 <= n <= 16384 and three results");
  cudaStream_t s = nullptr;
  pa::CholLookahead la;
  double* A = nullptr;
  int* info = nullptr;
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&la.aux, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&la.ev_panel, cudaEventDisableTiming);
  for (auto& v : la.ev_rest)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
  const size_t nn = static_cast<size_t>(n) * n;
  if (e == cudaSuccess) e = cudaMalloc(&A, sizeof(double) * (nn + pa::linalg_workspace_doubles(n)));
  if (e == cudaSuccess) e = cudaMalloc(&info, sizeof(int));
  if (e == cudaSuccess) e = cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed);
  Order o;
  if (e == cudaSuccess) {
    pa::cholesky_lower(A, n, info, A + nn, s, &la);
    e = cudaStreamEndCapture(s, &graph);  // fails when the second stream is not joined
  }
  if (e == cudaSuccess) e = read_order(graph, n, &o);
  if (graph) cudaGraphDestroy(graph);
  cudaFree(A);
  cudaFree(info);
  if (la.ev_panel) cudaEventDestroy(la.ev_panel);
  for (auto& v : la.ev_rest)
    if (v) cudaEventDestroy(v);
  if (la.aux) cudaStreamDestroy(la.aux);
  if (s) cudaStreamDestroy(s);
  if (e != cudaSuccess) return pa::set_error(PA_ERR_CUDA, std::string("pa_cholesky_order_check: ") + cudaGetErrorString(e));
  *missing = o.missing;
  *apart = o.apart;
  *pairs = o.pairs;
  return PA_OK;
}
