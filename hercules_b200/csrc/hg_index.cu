// hg_index.cu -- host side of the B200 Hercules index: tree construction with
// GPU-side routing and envelopes, the reference's on-disk format, and the
// query orchestration behind the C ABI of include/hercules_gpu.h.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <string>
#include <thread>
#include <map>
#include <vector>

#include "hg_arith.cuh"
#include "hg_breakpoints.h"
#include "hg_gen.cuh"
#include "hg_internal.h"
#include "hg_kernels.h"

using hg::Node;

// Launch geometry of the leaf scan.

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------

static thread_local char g_last_error[512] = "";

static hg_status set_error(hg_status s, const char* what) {
  snprintf(g_last_error, sizeof g_last_error, "%s", what);
  return s;
}

void hg_record_error(const char* msg) { set_error(HG_OK, msg); }

static hg_status cuda_fail(cudaError_t e, const char* where) {
  cudaGetLastError();  // reported here: not again by the next call's first launch
  char buf[512];
  snprintf(buf, sizeof buf, "%s: %s", where, cudaGetErrorString(e));
  return set_error(e == cudaErrorMemoryAllocation ? HG_ERR_NOMEM : HG_ERR_CUDA, buf);
}

#define CK(call)                                          \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return cuda_fail(e_, #call);   \
  } while (0)

#define HCK(call)                    \
  do {                               \
    hg_status s_ = (call);           \
    if (s_ != HG_OK) return s_;      \
  } while (0)

template <class T>
static cudaError_t dalloc(T** p, size_t count) {
  *p = nullptr;
  if (count == 0) count = 1;
  return cudaMalloc((void**)p, sizeof(T) * count);
}

template <class T>
static void dfree(T*& p) {
  if (p) cudaFree((void*)p);
  p = nullptr;
}

// ---------------------------------------------------------------------------
// tree algorithm (host, float arithmetic compiled with -ffp-contract=off)
// ---------------------------------------------------------------------------

namespace {

int seg_start(const std::vector<short>& p, int i) { return i == 0 ? 0 : p[i - 1]; }
int seg_len(const std::vector<short>& p, int i) { return i == 0 ? p[0] : p[i] - p[i - 1]; }

// calc_hs_split_points, hercules_node_split.c:371-396 (min_length = 1)
std::vector<short> hs_points_of(const std::vector<short>& points) {
  std::vector<short> hs;
  for (size_t i = 0; i < points.size(); ++i) {
    short length = points[i];
    if (i > 0) length = (short)(points[i] - points[i - 1]);
    if (length >= 2) {
      int start = i > 0 ? points[i - 1] : 0;
      hs.push_back((short)(start + (length / 2)));
    }
    hs.push_back(points[i]);
  }
  return hs;
}

// create_hercules_node_filename, hercules_node.c:441-486
std::string filename_of(const Node& n, const Node* parent) {
  char buf[256];
  int l = snprintf(buf, sizeof buf, "%02d", (int)n.points.size());
  if (n.level) {
    l += snprintf(buf + l, sizeof buf - l, "%s", n.is_left ? "_L" : "_R");
    l += snprintf(buf + l, sizeof buf - l, "%s", parent->split_idx ? "_1" : "_0");
    l += snprintf(buf + l, sizeof buf - l, "_(%d,%d,%g)", parent->split_from, parent->split_to,
                  (double)parent->split_value);
  }
  snprintf(buf + l, sizeof buf - l, "_%d", n.level);
  return buf;
}

void init_sketch(std::vector<float>& s, size_t nseg) {
  s.assign(4 * nseg, 0.0f);
  for (size_t i = 0; i < nseg; ++i) {
    s[4 * i + 0] = -FLT_MAX;
    s[4 * i + 1] = FLT_MAX;
    s[4 * i + 2] = -FLT_MAX;
    s[4 * i + 3] = FLT_MAX;
  }
}

Node make_leaf(const std::vector<short>& points) {
  Node n;
  n.points = points;
  n.hs_points = hs_points_of(points);
  init_sketch(n.sk, points.size());
  return n;
}

// range_calc, hercules_node_split.c:337-345
float range_calc(const float* ind, int len) {
  float mean_width = ind[0] - ind[1];
  float stdev_upper = ind[2];
  return (float)len * (mean_width * mean_width + stdev_upper * stdev_upper);
}

// mean/stdev split policies (hercules_node_split.c:22-71) for one segment
// sketch: the splitting benefit QoS(N) - mean(QoS children) and the value.
float policy_diff(const float* ind, int len, int policy, float* value) {
  float c0[4], c1[4];
  memcpy(c0, ind, sizeof c0);
  memcpy(c1, ind, sizeof c1);
  float v;
  if (policy == 0) {
    v = (ind[0] + ind[1]) / 2;
    c0[1] = v;
    c1[0] = v;
  } else {
    v = (ind[2] + ind[3]) / 2;
    c0[2] = v;
    c1[3] = v;
  }
  *value = v;
  float r0 = range_calc(c0, len), r1 = range_calc(c1, len);
  float mean = 0.0f;  // calc_mean, calc_utils.c:165-188
  mean = mean + r0;
  mean = mean + r1;
  mean = mean / (float)2;
  return range_calc(ind, len) - mean;
}

// The split decision of hercules_index_split_node (hercules_node_split.c:
// 1043-1252): best vertical policy, then horizontal candidates that must
// beat twice the best vertical benefit.  Returns the child segment ends.
std::vector<short> choose_split(Node& n, const std::vector<float>& hs_sk) {
  float max_diff = -FLT_MAX;
  int hs_split_point = -1;
  short from = 0, to = 0;
  int idx = 0;
  float value = 0.0f;
  for (size_t i = 0; i < n.points.size(); ++i) {
    int len = seg_len(n.points, (int)i);
    for (int j = 0; j < 2; ++j) {
      float v;
      float diff = policy_diff(&n.sk[4 * i], len, j, &v);
      if (diff > max_diff) {
        max_diff = diff;
        from = (short)seg_start(n.points, (int)i);
        to = n.points[i];
        idx = j;
        value = v;
      }
    }
  }
  max_diff = max_diff * 2;
  for (size_t i = 0; i < n.hs_points.size(); ++i) {
    int len = seg_len(n.hs_points, (int)i);
    for (int j = 0; j < 2; ++j) {
      float v;
      float diff = policy_diff(&hs_sk[4 * i], len, j, &v);
      if (diff > max_diff) {
        max_diff = diff;
        from = (short)seg_start(n.hs_points, (int)i);
        to = n.hs_points[i];
        idx = j;
        value = v;
        // get_hs_split_point, hercules_node_split.c:296-313
        bool found = std::find(n.points.begin(), n.points.end(), to) != n.points.end();
        hs_split_point = found ? from : to;
      }
    }
  }
  n.split_from = from;
  n.split_to = to;
  n.split_idx = idx;
  n.split_value = value;
  std::vector<short> cp = n.points;
  if (hs_split_point >= 0) {
    cp.push_back((short)hs_split_point);
    std::stable_sort(cp.begin(), cp.end());
  }
  return cp;
}

// Sketch keys (order-preserving ints, as the kernel writes them) to the
// envelope of node_segment_sketch_update_sketch_parallel: fmaxf/fminf of
// the initial -FLT_MAX / FLT_MAX with the members' extremes.
float key_to_float(int k) {
  int b = k >= 0 ? k : k ^ 0x7fffffff;
  float f;
  memcpy(&f, &b, 4);
  return f;
}

void keys_to_sketch(const int* keys, size_t nseg, float* sk) {
  for (size_t i = 0; i < nseg; ++i) {
    const int* k = keys + 4 * i;
    sk[4 * i + 0] = k[0] == INT_MIN ? -FLT_MAX : fmaxf(-FLT_MAX, key_to_float(k[0]));
    sk[4 * i + 1] = k[1] == INT_MAX ? FLT_MAX : fminf(FLT_MAX, key_to_float(k[1]));
    sk[4 * i + 2] = k[2] == INT_MIN ? -FLT_MAX : fmaxf(-FLT_MAX, key_to_float(k[2]));
    sk[4 * i + 3] = k[3] == INT_MAX ? FLT_MAX : fminf(FLT_MAX, key_to_float(k[3]));
  }
}

// update_node_ancestors_statistics_for_non_split_segments,
// hercules_node.c:613-657: with split_segment = -1 (never set by the
// parallel build) segment i of a parent is merged with segment i of the child.
void merge_ancestors(std::vector<Node>& nodes, int leaf) {
  int cn = leaf, cp = nodes[leaf].parent;
  while (cp >= 0) {
    Node& p = nodes[cp];
    const Node& c = nodes[cn];
    for (size_t i = 0; i < p.points.size(); ++i) {
      p.sk[4 * i + 0] = fmaxf(p.sk[4 * i + 0], c.sk[4 * i + 0]);
      p.sk[4 * i + 1] = fminf(p.sk[4 * i + 1], c.sk[4 * i + 1]);
      p.sk[4 * i + 2] = fmaxf(p.sk[4 * i + 2], c.sk[4 * i + 2]);
      p.sk[4 * i + 3] = fminf(p.sk[4 * i + 3], c.sk[4 * i + 3]);
    }
    cn = cp;
    cp = p.parent;
  }
}

void collect_leaves(const std::vector<Node>& nodes, int n, std::vector<int>& out) {
  // iterative DFS, left first
  std::vector<int> st{n};
  while (!st.empty()) {
    int x = st.back();
    st.pop_back();
    if (nodes[x].is_leaf) out.push_back(x);
    else {
      st.push_back(nodes[x].right);
      st.push_back(nodes[x].left);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// device index assembly
// ---------------------------------------------------------------------------

static void drop_graphs(hg::BatchScratch& b) {
  for (cudaGraphExec_t& g : b.graph) {
    if (g) cudaGraphExecDestroy(g);
    g = nullptr;
  }
}

static void free_scratch(hg_index* ix) {
  hg::QueryScratch& s = ix->s;
  dfree(s.lb);
  dfree(s.approx_leaf);
  dfree(s.cand);
  dfree(s.cand_lb);
  dfree(s.cand_count);
  dfree(s.unit_prefix);
  dfree(s.row_prefix);
  dfree(s.group_q);
  dfree(s.group_row);
  dfree(s.counters);
  dfree(s.bound);
  dfree(s.kslots);
  dfree(s.parts);
  dfree(s.part_count);
  dfree(s.topk);
  dfree(s.topk_count);
  dfree(s.sax_tab);
  dfree(s.sort_keys);
  dfree(s.stats);
  s.err = nullptr;  // in stats
  dfree(s.actl);
  s.slots = 0;
}

static void free_lists(hg_index* ix) {
  dfree(ix->s.list);
  ix->s.list_slots = 0;
}

static void free_batch_scratch(hg::BatchScratch& b) {
  dfree(b.qbf);
  dfree(b.qmeta);
  dfree(b.qperm);
  dfree(b.approx);
  dfree(b.kq);
  dfree(b.slots);
  dfree(b.items);
  dfree(b.bm);
  dfree(b.bound);
  dfree(b.init);
  dfree(b.init_cnt);
  dfree(b.bucket);
  dfree(b.bucket_cnt);
  dfree(b.pairs);
  dfree(b.ok);
  dfree(b.ctl);
  dfree(b.qlist);
  dfree(b.seg_rows);
  dfree(b.seg_prefix);
  dfree(b.qbound);
  dfree(b.parts);
  dfree(b.part_cnt);
  dfree(b.qlist2);
  dfree(b.qin);
  dfree(b.out_dist);
  dfree(b.out_id);
  dfree(b.leaf_plan);
  dfree(b.group_cnt);
  dfree(b.leaf_qoff);
  dfree(b.leaf_qcnt);
  dfree(b.item_off);
  drop_graphs(b);
  dfree(b.leaf_cnt);
  dfree(b.leaf_q);
  dfree(b.leaf_poff);
  dfree(b.leaf_ioff);
  dfree(b.panel_list);
  dfree(b.panel_bf);
  dfree(b.items3);
  dfree(b.useg_start);
  dfree(b.useg_end);
  dfree(b.seg_uid);
  dfree(b.segstats);
  b = hg::BatchScratch{};
}

static void free_device(hg_index* ix) {
  hg::DeviceIndex& d = ix->d;
  dfree(d.rows);
  dfree(d.rows_rm);
  dfree(d.ids);
  dfree(d.sax);
  dfree(d.bp);
  dfree(d.leaf_start);
  dfree(d.leaf_size);
  dfree(d.leaf_seg_off);
  dfree(d.leaf_points);
  dfree(d.leaf_sk);
  dfree(d.nodes);
  free_scratch(ix);
  free_lists(ix);
  dfree(ix->io.q);
  dfree(ix->io.out);
  ix->io = hg::HostIo{};
  for (cudaEvent_t& e : ix->ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  hg::BatchData& bd = ix->bd;
  dfree(bd.xbf);
  dfree(bd.xmeta);
  dfree(bd.tile_meta);
  free_batch_scratch(ix->bs);
}

// Routing tree in the final encoding: internal nodes renumbered densely,
// leaf children as ~leaf_index (DFS).
static std::vector<hg::DNode> routing_nodes(const hg_index* ix, int* root) {
  std::vector<int> dense(ix->nodes.size(), -1);
  int cnt = 0;
  for (size_t i = 0; i < ix->nodes.size(); ++i)
    if (!ix->nodes[i].is_leaf) dense[i] = cnt++;
  std::vector<hg::DNode> out(cnt > 0 ? cnt : 1);
  auto enc = [&](int nid) { return ix->nodes[nid].is_leaf ? ~ix->nodes[nid].leaf_index : dense[nid]; };
  for (size_t i = 0; i < ix->nodes.size(); ++i) {
    const Node& n = ix->nodes[i];
    if (n.is_leaf) continue;
    hg::DNode& d = out[dense[i]];
    d.left = enc(n.left);
    d.right = enc(n.right);
    d.value = n.split_value;
    d.from = n.split_from;
    d.to = n.split_to;
    d.idx = n.split_idx;
    d.pad = 0;
  }
  *root = enc(0);
  return out;
}

// Leaf tables and routing tree to the device (rows, ids, sax already there).
static hg_status upload_tables(hg_index* ix) {
  hg::DeviceIndex& d = ix->d;
  const size_t nl = ix->leaves.size();
  std::vector<uint64_t> start(nl);
  std::vector<uint32_t> size(nl);
  std::vector<int> off(nl + 1, 0);
  std::vector<short> pts;
  std::vector<float> sk;
  int max_seg = 0;
  for (size_t i = 0; i < nl; ++i) {
    const Node& n = ix->nodes[ix->leaves[i]];
    start[i] = n.file_pos;
    size[i] = n.node_size;
    off[i + 1] = off[i] + (int)n.points.size();
    pts.insert(pts.end(), n.points.begin(), n.points.end());
    sk.insert(sk.end(), n.sk.begin(), n.sk.end());
    max_seg = std::max(max_seg, (int)n.points.size());
  }
  ix->max_seg = max_seg;
  CK(dalloc(&d.leaf_start, nl));
  CK(dalloc(&d.leaf_size, nl));
  CK(dalloc(&d.leaf_seg_off, nl + 1));
  CK(dalloc(&d.leaf_points, pts.size()));
  CK(dalloc(&d.leaf_sk, sk.size()));
  CK(cudaMemcpy(d.leaf_start, start.data(), sizeof(uint64_t) * nl, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(d.leaf_size, size.data(), sizeof(uint32_t) * nl, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(d.leaf_seg_off, off.data(), sizeof(int) * (nl + 1), cudaMemcpyHostToDevice));
  if (!pts.empty()) CK(cudaMemcpy(d.leaf_points, pts.data(), sizeof(short) * pts.size(), cudaMemcpyHostToDevice));
  if (!sk.empty()) CK(cudaMemcpy(d.leaf_sk, sk.data(), sizeof(float) * sk.size(), cudaMemcpyHostToDevice));
  int root;
  std::vector<hg::DNode> rn = routing_nodes(ix, &root);
  CK(dalloc(&d.nodes, rn.size()));
  CK(cudaMemcpy(d.nodes, rn.data(), sizeof(hg::DNode) * rn.size(), cudaMemcpyHostToDevice));
  d.root = root;
  if (!d.bp) {
    CK(dalloc(&d.bp, 256));
    CK(cudaMemcpy(d.bp, kHgBreakpoints, sizeof(float) * 255, cudaMemcpyHostToDevice));
  }
  return HG_OK;
}

// ---------------------------------------------------------------------------
// build
// ---------------------------------------------------------------------------

namespace {

// The tree grows on the host, the rows stay on the device: node_of holds the
// node of every row routed so far (a leaf's members in insertion order are its
// rows in ascending order, as rows are inserted and redistributed in order).
// A window of rows is routed through the tree of the moment and the host
// counts the rows into their leaves.  A leaf that fills up waits for its
// split, and the window's later rows of that leaf wait with it; the other
// leaves do not depend on it, so the count goes on, and at the window's end
// all waiting leaves split together, in two device round trips (envelopes of
// the members, then their redistribution, which also moves the waiting rows).
// The waiting rows are counted again, until none waits.  The tree is the one
// that splits one at a time give.  Splitting one leaf at a time and routing
// the rest of the window again after it, with the member lists on the host,
// took 72 to 81 ms for 1M x 256, leaf 10,000 (193 leaves; 24 ms of it routing),
// and 1.35 to 1.41 s for 1M x 64, leaf 200 (8,468 leaves); this takes 20 to 21 and
// 52 to 63 ms (medians of three processes of 25 builds each; the rest is host
// memory management, and single builds take up to 58 ms where that is slow).
struct BuildCtx {
  hg_index* ix;
  const float* X;  // device, n x L row-major, original order
  cudaStream_t st;
  // device build scratch
  hg::DNode* d_tree = nullptr;
  size_t tree_cap = 0;
  int* d_node_of = nullptr;       // n
  uint32_t* d_list = nullptr;     // n: rows of the leaves being split
  uint32_t* d_count = nullptr;    // members collected and sent left per leaf, later rows
  size_t count_cap = 0;
  int* d_keys = nullptr;
  size_t keys_cap = 0;
  unsigned char* d_round = nullptr;  // tables of a round of splits
  size_t round_cap = 0;
  std::vector<hg::DNode> h_tree;  // node id -> routing entry (internal nodes)
  enum State : uint32_t { kLeaf, kWaiting, kInternal };
  struct Count {
    uint32_t rows = 0;  // of the leaf (an internal node: when it split)
    State state = kLeaf;
  };
  std::vector<Count> fill;        // by node
  std::vector<int> win;           // node of each row of the window
  bool tree_changed = true;
  int root_enc = ~0;
  // windows double with the rows inserted, so a leaf splits about once per
  // window; the largest bounds the rows counted again
  static constexpr uint32_t kWindowMin = 65536, kWindowMax = 262144;
  static constexpr int kMaxSegs = 4096;
  struct Full {
    int nid;
    uint32_t last;  // the row that filled the leaf
  };

  ~BuildCtx() {
    dfree(d_tree);
    dfree(d_node_of);
    dfree(d_list);
    dfree(d_count);
    dfree(d_keys);
    dfree(d_round);
  }

  template <class T>
  hg_status grow(T** p, size_t* cap, size_t want) {
    if (want <= *cap) return HG_OK;
    CK(cudaStreamSynchronize(st));
    dfree(*p);
    *cap = 0;
    CK(dalloc(p, 2 * want));
    *cap = 2 * want;
    return HG_OK;
  }

  // During the build a leaf child is encoded ~node_id.
  hg_status sync_tree() {
    if (!tree_changed) return HG_OK;
    HCK(grow(&d_tree, &tree_cap, std::max<size_t>(h_tree.size(), 512)));
    CK(cudaMemcpyAsync(d_tree, h_tree.data(), sizeof(hg::DNode) * h_tree.size(), cudaMemcpyHostToDevice, st));
    tree_changed = false;
    return HG_OK;
  }

  hg::Tree tree() const { return hg::Tree{d_tree, root_enc}; }

  // hercules_index_split_node (hercules_node_split.c:1043-1345) for each full
  // leaf; the rows below `end` are routed, `later` of them wait, and win (whose
  // first row is c) is brought up to date from position `from` on
  hg_status split(const std::vector<Full>& full, uint64_t c, uint64_t end, uint64_t later, uint32_t from) {
    std::vector<Node>& nodes = ix->nodes;
    const size_t P = full.size();
    // one upload: list start, slot of every node, size, last row and segments
    // (vertical, then horizontal candidates) of each leaf
    std::vector<int> seg_off(P + 1, 0);
    uint64_t members = 0;
    hg::SketchArgs a{};
    for (size_t p = 0; p < P; ++p) {
      const Node& n = nodes[full[p].nid];
      const int ns = (int)(n.points.size() + n.hs_points.size());
      if (ns > kMaxSegs) return set_error(HG_ERR_LIMIT, "too many EAPCA segments in one node");
      seg_off[p + 1] = seg_off[p] + ns;
      a.max_segs = std::max(a.max_segs, ns);
      a.max_size = std::max(a.max_size, fill[full[p].nid].rows);
    }
    const size_t T = (size_t)seg_off[P], N = nodes.size();
    const size_t o_start = 0, o_slot = o_start + 8 * P, o_size = o_slot + 4 * N, o_last = o_size + 4 * P,
                 o_off = o_last + 4 * P, o_seg = o_off + 4 * (P + 1), bytes = (o_seg + 4 * T + 7) & ~(size_t)7;
    const size_t o_split = bytes;  // the policies follow, written after the envelopes are known
    std::vector<unsigned char> h(bytes);
    uint64_t* start = reinterpret_cast<uint64_t*>(h.data() + o_start);
    int* slot = reinterpret_cast<int*>(h.data() + o_slot);
    uint32_t* size = reinterpret_cast<uint32_t*>(h.data() + o_size);
    uint32_t* last = reinterpret_cast<uint32_t*>(h.data() + o_last);
    short* seg = reinterpret_cast<short*>(h.data() + o_seg);
    std::fill(slot, slot + N, -1);
    memcpy(h.data() + o_off, seg_off.data(), 4 * (P + 1));
    for (size_t p = 0; p < P; ++p) {
      const Node& n = nodes[full[p].nid];
      start[p] = members;
      slot[full[p].nid] = (int)p;
      size[p] = fill[full[p].nid].rows;
      last[p] = full[p].last;
      members += size[p];
      size_t t = (size_t)seg_off[p];
      for (const std::vector<short>* pts : {&n.points, &n.hs_points})
        for (size_t i = 0; i < pts->size(); ++i, ++t) {
          seg[t] = (short)seg_start(*pts, (int)i);
          seg[T + t] = (*pts)[i];
        }
    }
    HCK(grow(&d_round, &round_cap, bytes + sizeof(hg::SplitPolicy) * P));
    HCK(grow(&d_count, &count_cap, 2 * P + 1));
    HCK(grow(&d_keys, &keys_cap, 4 * T));
    uint32_t *d_members = d_count, *d_left = d_count + P, *d_later = d_count + 2 * P;
    const int* d_slot = reinterpret_cast<int*>(d_round + o_slot);
    CK(cudaMemcpyAsync(d_round, h.data(), bytes, cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(d_count, 0, sizeof(uint32_t) * (2 * P + 1), st));
    a.X = X;
    a.L = (int)ix->L;
    a.members = d_list;
    a.ngroups = (int)P;
    a.start = reinterpret_cast<uint64_t*>(d_round + o_start);
    a.size = reinterpret_cast<uint32_t*>(d_round + o_size);
    a.seg_off = reinterpret_cast<int*>(d_round + o_off);
    a.seg_from = reinterpret_cast<short*>(d_round + o_seg);
    a.seg_to = a.seg_from + T;
    a.keys = d_keys;
    CK(hg::launch_collect_members(d_node_of, end, d_slot, a.start, reinterpret_cast<uint32_t*>(d_round + o_last), members,
                                  d_list, d_members, d_later, d_keys, (int)T, st));
    CK(hg::launch_sketch(a, st));
    std::vector<int> keys(4 * T);
    CK(cudaMemcpyAsync(keys.data(), d_keys, sizeof(int) * 4 * T, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<hg::SplitPolicy> pol(P);
    std::vector<float> hs_sk;
    for (size_t p = 0; p < P; ++p) {
      const int nid = full[p].nid;
      const size_t nv = nodes[nid].points.size(), nh = nodes[nid].hs_points.size();
      const int* k = &keys[4 * (size_t)seg_off[p]];
      hs_sk.resize(4 * nh);
      nodes[nid].sk.resize(4 * nv);
      keys_to_sketch(k, nv, nodes[nid].sk.data());
      keys_to_sketch(k + 4 * nv, nh, hs_sk.data());
      std::vector<short> cp = choose_split(nodes[nid], hs_sk);
      // children (split_node_create_children, hercules_node_split.c:197-262)
      Node l = make_leaf(cp), r = make_leaf(cp);
      l.parent = r.parent = nid;
      l.level = r.level = nodes[nid].level + 1;
      l.is_left = true;
      l.filename = filename_of(l, &nodes[nid]);
      r.filename = filename_of(r, &nodes[nid]);
      const int lid = (int)nodes.size(), rid = lid + 1;
      nodes.push_back(std::move(l));
      nodes.push_back(std::move(r));
      Node& n = nodes[nid];
      n.left = lid;
      n.right = rid;
      n.is_leaf = false;
      n.node_size = fill[nid].rows;
      pol[p] = hg::SplitPolicy{n.split_value, lid, rid, n.split_from, n.split_to, n.split_idx};
      // routing entries: this node becomes internal, its parent points to it
      if (h_tree.size() < nodes.size()) h_tree.resize(nodes.size());
      h_tree[nid] = hg::DNode{~lid, ~rid, n.split_value, n.split_from, n.split_to, n.split_idx, 0};
      if (n.parent < 0) root_enc = nid;
      else {
        hg::DNode& d = h_tree[n.parent];
        if (d.left == ~nid) d.left = nid;
        else d.right = nid;
      }
    }
    tree_changed = true;
    hg::SplitPolicy* d_pol = reinterpret_cast<hg::SplitPolicy*>(d_round + o_split);
    CK(cudaMemcpyAsync(d_pol, pol.data(), sizeof(hg::SplitPolicy) * P, cudaMemcpyHostToDevice, st));
    CK(hg::launch_split_members(X, (int)ix->L, d_node_of, d_list, members, d_later, later, d_slot, d_pol, d_left, st));
    std::vector<uint32_t> cnt(2 * P + 1);
    CK(cudaMemcpyAsync(cnt.data(), d_count, sizeof(uint32_t) * cnt.size(), cudaMemcpyDeviceToHost, st));
    if (later)
      CK(cudaMemcpyAsync(win.data() + from, d_node_of + c + from, sizeof(int) * (end - c - from), cudaMemcpyDeviceToHost,
                         st));
    CK(cudaStreamSynchronize(st));
    fill.resize(nodes.size());
    for (size_t p = 0; p < P; ++p) {
      const uint32_t left = cnt[P + p];
      if (cnt[p] != size[p] || left > size[p])
        return set_error(HG_ERR_CUDA, "internal: a split lost or invented rows");
      fill[full[p].nid].state = kInternal;
      fill[pol[p].left].rows = left;
      fill[pol[p].right].rows = size[p] - left;
    }
    if (cnt[2 * P] != later) return set_error(HG_ERR_CUDA, "internal: a split lost or invented rows");
    return HG_OK;
  }

  hg_status run() {
    std::vector<Node>& nodes = ix->nodes;
    const uint64_t n = ix->n;
    const uint32_t S = ix->leaf_size;
    CK(dalloc(&d_node_of, n));
    CK(dalloc(&d_list, n));
    h_tree.resize(1);
    fill.resize(1);
    std::vector<Full> full;
    std::vector<uint32_t> waiting, again;  // window positions, ascending
    for (uint64_t c = 0; c < n;) {
      const uint64_t grown = std::min<uint64_t>(kWindowMax, std::max<uint64_t>(kWindowMin, c));
      const uint32_t w = (uint32_t)std::min<uint64_t>(grown, n - c);
      win.resize(w);
      HCK(sync_tree());
      CK(hg::launch_route_rows(X, (int)ix->L, c, w, tree(), d_node_of + c, st));
      CK(cudaMemcpyAsync(win.data(), d_node_of + c, sizeof(int) * w, cudaMemcpyDeviceToHost, st));
      CK(cudaStreamSynchronize(st));
      bool bad = false;
      auto insert = [&](uint32_t j) {
        const uint32_t nid = (uint32_t)win[j];
        if (nid >= fill.size()) {
          bad = true;
          return;
        }
        Count& leaf = fill[nid];
        if (leaf.state != kLeaf) {
          if (leaf.state == kWaiting) waiting.push_back(j);
          else bad = true;
        } else if (++leaf.rows >= S) {
          leaf.state = kWaiting;
          full.push_back(Full{(int)nid, (uint32_t)(c + j)});
        }
      };
      for (uint32_t j = 0; j < w; ++j) insert(j);
      while (!full.empty() && !bad) {
        HCK(split(full, c, c + w, waiting.size(), waiting.empty() ? w : waiting.front()));
        full.clear();
        again.swap(waiting);
        waiting.clear();
        for (uint32_t j : again) insert(j);
      }
      if (bad) return set_error(HG_ERR_CUDA, "internal: routing returned a node that is not a leaf");
      c += w;
    }
    for (size_t i = 0; i < nodes.size(); ++i)
      if (nodes[i].is_leaf) nodes[i].node_size = fill[i].rows;
    return HG_OK;
  }
};

}  // namespace

// Leaf order, file positions, leaf envelopes, the leaf-ordered tiles, iSAX
// words and the merged internal envelopes of the written index.
static hg_status finalize_build(hg_index* ix, const float* X, cudaStream_t st, const BuildCtx& ctx) {
  std::vector<Node>& nodes = ix->nodes;
  ix->leaves.clear();
  collect_leaves(nodes, 0, ix->leaves);
  const size_t nl = ix->leaves.size();
  uint64_t pos = 0;
  std::vector<uint64_t> at(nodes.size(), 0);  // next leaf-ordered row of each leaf
  for (size_t i = 0; i < nl; ++i) {
    Node& lf = nodes[ix->leaves[i]];
    lf.leaf_index = (int)i;
    lf.file_pos = pos;
    at[ix->leaves[i]] = pos;
    pos += lf.node_size;
  }
  if (pos != ix->n) return set_error(HG_ERR_ARG, "internal: leaf sizes do not add up");
  // leaf order: the rows of each leaf in ascending order
  std::vector<uint32_t> perm(ix->n);
  {
    std::vector<int> node_of(ix->n);
    CK(cudaMemcpyAsync(node_of.data(), ctx.d_node_of, sizeof(int) * ix->n, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (uint64_t r = 0; r < ix->n; ++r) perm[at[node_of[r]]++] = (uint32_t)r;
  }
  uint32_t* d_perm = ctx.d_list;
  CK(cudaMemcpyAsync(d_perm, perm.data(), sizeof(uint32_t) * ix->n, cudaMemcpyHostToDevice, st));
  // leaf-ordered rows, ids, iSAX words
  hg::DeviceIndex& d = ix->d;
  CK(dalloc(&d.rows, (size_t)ix->n * ix->L));
  CK(hg::launch_gather_rows(X, ix->L, d_perm, ix->n, d.rows, st));
  CK(dalloc(&d.ids, ix->n));
  CK(hg::launch_widen_ids(d_perm, ix->n, d.ids, st));
  CK(dalloc(&d.bp, 256));
  CK(cudaMemcpyAsync(d.bp, kHgBreakpoints, sizeof(float) * 255, cudaMemcpyHostToDevice, st));
  // padded to whole 32-row units: the LB_SAX filter bulk-copies whole units
  CK(dalloc(&d.sax, (size_t)((ix->n + 31) & ~31ull) * 16));
  CK(hg::launch_sax_rows(d.rows, ix->L, ix->n, d.bp, d.sax, st));
  // leaf envelopes: vertical sketches over each leaf's rows, all leaves in one launch
  std::vector<uint64_t> start(nl);
  std::vector<uint32_t> size(nl);
  std::vector<int> koff(nl + 1, 0);
  hg::SketchArgs a{};
  for (size_t i = 0; i < nl; ++i) {
    const Node& lf = nodes[ix->leaves[i]];
    start[i] = lf.file_pos;
    size[i] = lf.node_size;
    koff[i + 1] = koff[i] + (int)lf.points.size();
    a.max_segs = std::max(a.max_segs, (int)lf.points.size());
    a.max_size = std::max(a.max_size, lf.node_size);
  }
  const size_t total_segs = (size_t)koff[nl];
  std::vector<short> seg(2 * total_segs);
  std::vector<int> keys(4 * total_segs);
  for (size_t i = 0; i < nl; ++i) {
    const Node& lf = nodes[ix->leaves[i]];
    for (size_t s = 0; s < lf.points.size(); ++s) {
      seg[koff[i] + s] = (short)seg_start(lf.points, (int)s);
      seg[total_segs + koff[i] + s] = lf.points[s];
    }
  }
  for (size_t i = 0; i < keys.size(); ++i) keys[i] = (i & 1) ? INT_MAX : INT_MIN;
  int *d_keys = nullptr, *d_off = nullptr;
  short* d_seg = nullptr;
  uint64_t* d_start = nullptr;
  uint32_t* d_size = nullptr;
  auto release = [](void* p) { cudaFree(p); };
  using Guard = std::unique_ptr<void, void (*)(void*)>;
  CK(dalloc(&d_keys, keys.size()));
  Guard g1(d_keys, release);
  CK(dalloc(&d_off, nl + 1));
  Guard g2(d_off, release);
  CK(dalloc(&d_seg, seg.size()));
  Guard g3(d_seg, release);
  CK(dalloc(&d_start, nl));
  Guard g4(d_start, release);
  CK(dalloc(&d_size, nl));
  Guard g5(d_size, release);
  CK(cudaMemcpyAsync(d_keys, keys.data(), sizeof(int) * keys.size(), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(d_off, koff.data(), sizeof(int) * (nl + 1), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(d_seg, seg.data(), sizeof(short) * seg.size(), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(d_start, start.data(), sizeof(uint64_t) * nl, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(d_size, size.data(), sizeof(uint32_t) * nl, cudaMemcpyHostToDevice, st));
  a.X = d.rows;
  a.L = (int)ix->L;
  a.ngroups = (int)nl;
  a.start = d_start;
  a.size = d_size;
  a.seg_off = d_off;
  a.seg_from = d_seg;
  a.seg_to = d_seg + total_segs;
  a.keys = d_keys;
  CK(hg::launch_sketch(a, st));
  CK(cudaMemcpyAsync(keys.data(), d_keys, sizeof(int) * keys.size(), cudaMemcpyDeviceToHost, st));
  ix->ids.assign(perm.begin(), perm.end());
  ix->has_ids = true;
  CK(cudaStreamSynchronize(st));
  for (size_t i = 0; i < nl; ++i) {
    Node& lf = nodes[ix->leaves[i]];
    if (lf.node_size == 0) continue;  // an empty leaf keeps the initial envelope
    keys_to_sketch(&keys[4 * (size_t)koff[i]], lf.points.size(), lf.sk.data());
  }
  // internal envelopes as the sequential writer leaves them
  for (size_t i = 0; i < ix->leaves.size(); ++i) merge_ancestors(nodes, ix->leaves[i]);
  return upload_tables(ix);
}

static hg_status build_impl(const float* data, int on_device, uint64_t n, uint32_t L, uint32_t S, int device,
                            hg_index** out) {
  if (!out || !data || n == 0 || L == 0 || L % 16 != 0 || L > 32752 || S == 0)
    return set_error(HG_ERR_ARG, "hg_index_build: need data, n > 0, L a multiple of 16 (<= 32752), leaf size > 0");
  if (n > 0xffffffffull) return set_error(HG_ERR_LIMIT, "hg_index_build: at most 2^32-1 series");
  CK(cudaSetDevice(device));
  std::unique_ptr<hg_index> ix(new hg_index());
  ix->device = device;
  ix->L = L;
  ix->leaf_size = S;
  ix->n = n;
  CK(cudaStreamCreateWithFlags(&ix->stream, cudaStreamNonBlocking));
  const float* X = data;
  float* owned = nullptr;
  if (!on_device) {
    CK(dalloc(&owned, n * L));
    // staged copy from pageable memory in 256 MiB pieces
    const size_t piece = (256u << 20) / (sizeof(float) * L) * L;
    for (size_t o = 0; o < n * L; o += piece) {
      size_t cnt = std::min(piece, (size_t)(n * L - o));
      CK(cudaMemcpyAsync(owned + o, data + o, sizeof(float) * cnt, cudaMemcpyHostToDevice, ix->stream));
    }
    X = owned;
  }
  std::unique_ptr<float, void (*)(float*)> g(owned, [](float* p) {
    if (p) cudaFree(p);
  });
  // root (hercules_root_node_init, hercules_node.c:27-78): one segment [0, L)
  Node root = make_leaf(std::vector<short>{(short)L});
  root.filename = filename_of(root, nullptr);
  ix->nodes.push_back(std::move(root));
  hg_status s;
  {
    BuildCtx ctx;
    ctx.ix = ix.get();
    ctx.X = X;
    ctx.st = ix->stream;
    s = ctx.run();
    if (s == HG_OK) s = finalize_build(ix.get(), X, ix->stream, ctx);
  }
  if (s != HG_OK) {
    cudaStreamSynchronize(ix->stream);
    free_device(ix.get());
    cudaStreamDestroy(ix->stream);
    return s;
  }
  *out = ix.release();
  return HG_OK;
}

// ---------------------------------------------------------------------------
// on-disk format (App. A of the format: root.idx, leaves_raw.idx, leaves_sims.idx)
// ---------------------------------------------------------------------------

namespace {

struct Writer {
  FILE* f;
  bool ok = true;
  template <class T>
  void put(const T& v) { ok = ok && fwrite(&v, sizeof(T), 1, f) == 1; }
  void bytes(const void* p, size_t n) { ok = ok && (n == 0 || fwrite(p, 1, n, f) == n); }
};

// hercules_node_write, hercules_index.c:1967-2077
void write_node(const hg_index* ix, int nid, Writer& w) {
  const Node& n = ix->nodes[nid];
  w.put<uint8_t>(n.is_leaf ? 1 : 0);
  w.put<uint32_t>(n.level);
  if (!n.is_leaf) {
    write_node(ix, n.left, w);
    write_node(ix, n.right, w);
    w.put<uint32_t>(n.node_size);
    w.put<int16_t>(-1);  // split_segment, never set by the parallel build
    // struct node_split_policy (48 bytes, hercules_node_split.h:21-34): the
    // trailing padding and pointer bytes carry no information; zeros here.
    uint8_t pol[48];
    memset(pol, 0, sizeof pol);
    memcpy(pol + 0, &n.split_from, 2);
    memcpy(pol + 2, &n.split_to, 2);
    memcpy(pol + 4, &n.split_value, 4);
    memcpy(pol + 8, &n.split_idx, 4);
    memcpy(pol + 12, &n.split_idx, 4);
    memcpy(pol + 16, &n.split_value, 4);
    w.bytes(pol, 48);
  } else {
    w.put<uint32_t>(n.node_size);
    w.put<int32_t>((int32_t)n.filename.size());
    w.bytes(n.filename.data(), n.filename.size());
  }
  w.put<int16_t>((int16_t)n.points.size());
  w.bytes(n.points.data(), sizeof(short) * n.points.size());
  for (size_t i = 0; i < n.points.size(); ++i) {
    w.put<int32_t>(4);
    w.bytes(&n.sk[4 * i], 16);
  }
  if (n.is_leaf) w.put<uint64_t>(n.file_pos);
}

struct Reader {
  FILE* f;
  bool ok = true;
  template <class T>
  T get() {
    T v{};
    ok = ok && fread(&v, sizeof(T), 1, f) == 1;
    return v;
  }
  void bytes(void* p, size_t n) { ok = ok && (n == 0 || fread(p, 1, n, f) == n); }
};

// hercules_node_read, hercules_index.c:2188-2340
int read_node(hg_index* ix, Reader& r, int parent, int depth) {
  if (!r.ok || depth > 10000) return -1;
  const int nid = (int)ix->nodes.size();
  ix->nodes.emplace_back();
  const uint8_t is_leaf = r.get<uint8_t>();
  const uint32_t level = r.get<uint32_t>();
  ix->nodes[nid].parent = parent;
  ix->nodes[nid].level = level;
  ix->nodes[nid].is_leaf = is_leaf != 0;
  if (!is_leaf) {
    int l = read_node(ix, r, nid, depth + 1);
    int rr = read_node(ix, r, nid, depth + 1);
    if (l < 0 || rr < 0) return -1;
    Node& n = ix->nodes[nid];
    n.left = l;
    n.right = rr;
    ix->nodes[l].is_left = true;
    n.node_size = r.get<uint32_t>();
    (void)r.get<int16_t>();
    uint8_t pol[48];
    r.bytes(pol, 48);
    memcpy(&n.split_from, pol + 0, 2);
    memcpy(&n.split_to, pol + 2, 2);
    memcpy(&n.split_idx, pol + 12, 4);
    memcpy(&n.split_value, pol + 16, 4);
  } else {
    Node& n = ix->nodes[nid];
    n.node_size = r.get<uint32_t>();
    const int32_t len = r.get<int32_t>();
    if (len <= 0) {
      n.node_size = 0;  // a leaf written without a file name holds nothing
      return r.ok ? nid : -1;
    }
    if (len > 65536) return -1;
    n.filename.resize(len);
    r.bytes(&n.filename[0], len);
  }
  Node& n = ix->nodes[nid];
  const int16_t np = r.get<int16_t>();
  if (np < 0 || np > 32767) return -1;
  n.points.resize(np);
  r.bytes(n.points.data(), sizeof(short) * np);
  n.sk.resize(4 * np);
  for (int i = 0; i < np; ++i) {
    if (r.get<int32_t>() != 4) return -1;
    r.bytes(&n.sk[4 * i], 16);
  }
  if (n.is_leaf) n.file_pos = r.get<uint64_t>();
  return r.ok ? nid : -1;
}

std::string join(const char* dir, const char* name) {
  std::string s(dir);
  return s + name;
}

}  // namespace

static hg_status write_impl(hg_index* ix, const char* dir, double buffer_mb) {
  if (!ix || !dir) return set_error(HG_ERR_ARG, "hg_index_write: null argument");
  CK(cudaSetDevice(ix->device));
  FILE* f = fopen(join(dir, "root.idx").c_str(), "wb");
  FILE* raw = fopen(join(dir, "leaves_raw.idx").c_str(), "wb");
  FILE* sims = fopen(join(dir, "leaves_sims.idx").c_str(), "wb");
  FILE* idf = fopen(join(dir, "leaves_ids.idx").c_str(), "wb");
  auto close_all = [&]() {
    if (f) fclose(f);
    if (raw) fclose(raw);
    if (sims) fclose(sims);
    if (idf) fclose(idf);
  };
  if (!f || !raw || !sims || !idf) {
    close_all();
    return set_error(HG_ERR_IO, "hg_index_write: cannot create the index files");
  }
  // header (hercules_index.c:1671-1682)
  Writer w{f};
  w.put<uint64_t>((uint64_t)ix->leaves.size());
  w.put<double>(buffer_mb);
  w.put<uint32_t>(ix->L);
  w.put<uint32_t>(1u);
  w.put<int32_t>(16);
  w.put<int32_t>(8);
  w.put<uint32_t>(ix->leaf_size);
  w.put<int32_t>(1);
  w.put<int32_t>(1);
  write_node(ix, 0, w);
  // leaf-ordered raw rows (the HBM image) and iSAX words, in pieces
  const uint64_t piece = std::max<uint64_t>(1, (64u << 20) / (sizeof(float) * ix->L));
  std::vector<float> h_rm(piece * ix->L);
  std::vector<uint8_t> h_sax(piece * 16);
  bool ok = w.ok;
  for (uint64_t r0 = 0; r0 < ix->n && ok; r0 += piece) {
    const uint64_t cnt = std::min(piece, ix->n - r0);
    cudaError_t e = cudaMemcpyAsync(h_rm.data(), ix->d.rows + r0 * ix->L, sizeof(float) * cnt * ix->L,
                                    cudaMemcpyDeviceToHost, ix->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_sax.data(), ix->d.sax + r0 * 16, cnt * 16, cudaMemcpyDeviceToHost, ix->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
    if (e != cudaSuccess) {
      close_all();
      return cuda_fail(e, "hg_index_write");
    }
    ok = fwrite(h_rm.data(), sizeof(float) * ix->L, cnt, raw) == cnt && fwrite(h_sax.data(), 16, cnt, sims) == cnt;
  }
  std::vector<uint64_t> ids64(ix->n);
  for (uint64_t i = 0; i < ix->n; ++i) ids64[i] = ix->has_ids ? (uint64_t)ix->ids[i] : i;
  ok = ok && fwrite(ids64.data(), 8, ix->n, idf) == ix->n;
  close_all();
  return ok ? HG_OK : set_error(HG_ERR_IO, "hg_index_write: short write");
}

// The device half of hg_index_read: rows from the open leaves_raw.idx
// (closed here), ids, breakpoints, iSAX words and the tables.
static hg_status read_device_part(hg_index* ix, FILE* raw, const char* dir) {
  hg::DeviceIndex& d = ix->d;
  // leaves_raw.idx is the HBM image: copy it in pieces
  const uint64_t piece = std::max<uint64_t>(1, (64u << 20) / (sizeof(float) * ix->L));
  std::vector<float> h_rm(piece * ix->L);
  cudaError_t e = dalloc(&d.rows, (size_t)ix->n * ix->L);
  for (uint64_t r0 = 0; r0 < ix->n && e == cudaSuccess; r0 += piece) {
    const uint64_t cnt = std::min(piece, ix->n - r0);
    if (fread(h_rm.data(), sizeof(float) * ix->L, cnt, raw) != cnt) {
      fclose(raw);
      free_device(ix);
      return set_error(HG_ERR_IO, "hg_index_read: leaves_raw.idx is shorter than the leaves");
    }
    e = cudaMemcpy(d.rows + r0 * ix->L, h_rm.data(), sizeof(float) * cnt * ix->L, cudaMemcpyHostToDevice);
  }
  fclose(raw);
  if (e != cudaSuccess) {
    free_device(ix);
    return cuda_fail(e, "hg_index_read");
  }
  // dataset ids: leaves_ids.idx when present, else the row number
  ix->ids.resize(ix->n);
  FILE* idf = fopen(join(dir, "leaves_ids.idx").c_str(), "rb");
  ix->has_ids = false;
  if (idf) {
    std::vector<uint64_t> ids64(ix->n);
    if (fread(ids64.data(), 8, ix->n, idf) == ix->n) {
      for (uint64_t i = 0; i < ix->n; ++i) ix->ids[i] = (int64_t)ids64[i];
      ix->has_ids = true;
    }
    fclose(idf);
  }
  if (!ix->has_ids)
    for (uint64_t i = 0; i < ix->n; ++i) ix->ids[i] = (int64_t)i;
  CK(dalloc(&d.ids, ix->n));
  CK(cudaMemcpy(d.ids, ix->ids.data(), sizeof(int64_t) * ix->n, cudaMemcpyHostToDevice));
  CK(dalloc(&d.bp, 256));
  CK(cudaMemcpy(d.bp, kHgBreakpoints, sizeof(float) * 255, cudaMemcpyHostToDevice));
  // padded to whole 32-row units: the LB_SAX filter bulk-copies whole units
  CK(dalloc(&d.sax, (size_t)((ix->n + 31) & ~31ull) * 16));
  CK(hg::launch_sax_rows(d.rows, ix->L, ix->n, d.bp, d.sax, ix->stream));
  CK(cudaStreamSynchronize(ix->stream));
  HCK(upload_tables(ix));
  return HG_OK;
}

static hg_status read_impl(const char* dir, int device, hg_index** out) {
  if (!dir || !out) return set_error(HG_ERR_ARG, "hg_index_read: null argument");
  FILE* f = fopen(join(dir, "root.idx").c_str(), "rb");
  if (!f) return set_error(HG_ERR_IO, "hg_index_read: cannot open root.idx");
  std::unique_ptr<hg_index> ix(new hg_index());
  Reader r{f};
  const uint64_t nleaves_hdr = r.get<uint64_t>();
  ix->buffer_mb = r.get<double>();
  ix->L = r.get<uint32_t>();
  const uint32_t init_segments = r.get<uint32_t>();
  const int32_t paa = r.get<int32_t>();
  const int32_t card = r.get<int32_t>();
  ix->leaf_size = r.get<uint32_t>();
  const int32_t serial = r.get<int32_t>();
  (void)r.get<int32_t>();
  (void)init_segments;
  if (!r.ok || paa != 16 || card != 8 || ix->L == 0 || ix->L % 16 != 0 || !serial) {
    fclose(f);
    return set_error(HG_ERR_FORMAT, "hg_index_read: root.idx header is not a serial 16x8-bit Hercules index");
  }
  if (read_node(ix.get(), r, -1, 0) != 0) {
    fclose(f);
    return set_error(HG_ERR_FORMAT, "hg_index_read: malformed node records in root.idx");
  }
  fclose(f);
  collect_leaves(ix->nodes, 0, ix->leaves);
  uint64_t pos = 0;
  for (size_t i = 0; i < ix->leaves.size(); ++i) {
    Node& lf = ix->nodes[ix->leaves[i]];
    lf.leaf_index = (int)i;
    if (lf.node_size > 0 && lf.file_pos != pos)
      return set_error(HG_ERR_FORMAT, "hg_index_read: leaves are not stored in DFS order in leaves_raw.idx");
    lf.file_pos = pos;
    pos += lf.node_size;
  }
  (void)nleaves_hdr;
  ix->n = pos;
  ix->device = device;
  // the data file must hold every leaf's rows: checked before any device work
  FILE* raw = fopen(join(dir, "leaves_raw.idx").c_str(), "rb");
  if (!raw) return set_error(HG_ERR_IO, "hg_index_read: cannot open leaves_raw.idx");
  if (fseeko(raw, 0, SEEK_END) != 0 || (uint64_t)ftello(raw) < ix->n * ix->L * sizeof(float) ||
      fseeko(raw, 0, SEEK_SET) != 0) {
    fclose(raw);
    return set_error(HG_ERR_IO, "hg_index_read: leaves_raw.idx is shorter than the leaves");
  }
  {
    const cudaError_t e0 = cudaSetDevice(device);
    cudaError_t e1 = e0 == cudaSuccess ? cudaStreamCreateWithFlags(&ix->stream, cudaStreamNonBlocking) : e0;
    if (e1 != cudaSuccess) {
      fclose(raw);
      ix->stream = nullptr;
      return cuda_fail(e1, "hg_index_read");
    }
  }
  const hg_status st = read_device_part(ix.get(), raw, dir);
  if (st != HG_OK) {
    hg_index_destroy(ix.release());
    return st;
  }
  *out = ix.release();
  return HG_OK;
}

// ---------------------------------------------------------------------------
// queries
// ---------------------------------------------------------------------------

// Queries of a plain call that share each launch: up to kGroupSlots, fewer
// where the survivor lists (one entry per row and slot) would pass
// kGroupListBytes, but four of them whatever the collection's size.  A group
// hides the latency of a query's chain of small kernels behind the other
// queries' scans and fills the GPU from indexes whose leaves are too small to
// (per query, one at a time -> in groups: 1M x 256, leaf 100,000, k = 10:
// 139 -> 28 us; 100k x 16384: 480 -> 92 us; 8M x 256, k = 100: 800 -> 390 us).
// 4 GB of lists, 2% of the GPU's memory, hold 32 queries of 33M rows; with
// 512 MB 25M rows left groups of five (64 queries of 25M x 256: 63.0 ms, 54.9
// now, with LB_SAX 22.2 and 19.0; 32 of 30M x 96 15.2 and 13.6).  PSCAN, which
// reads no lists, keeps to the same groups: 32 queries of 80M x 64 take 60.0 ms
// in groups of 11, 61.5 together.
constexpr uint32_t kGroupSlots = 32;
constexpr uint64_t kGroupListBytes = 4ull << 30;
static uint32_t group_slots(const hg_index* ix, uint32_t nq) {
  const uint64_t by_list = std::max<uint64_t>(4, kGroupListBytes / (4 * std::max<uint64_t>(ix->n, 1)));
  const uint32_t most = (uint32_t)std::min<uint64_t>(kGroupSlots, by_list);
  const uint32_t groups = (nq + most - 1) / most;
  return groups ? (nq + groups - 1) / groups : 1;
}

static cudaError_t alloc_scratch(hg_index* ix, size_t slots) {
  hg::QueryScratch& s = ix->s;
  const size_t nl = ix->leaves.size();
  s.nparts = hg::sm_count(ix->device) * hg::ed_blocks_per_sm((int)ix->L);
  cudaError_t e = cudaSuccess;
  auto get = [&](auto** p, size_t count) {
    if (e == cudaSuccess) e = dalloc(p, count);
  };
  get(&s.lb, slots * nl);
  get(&s.counters, slots * 8);
  get(&s.approx_leaf, slots);
  get(&s.cand, slots * (nl + 1));
  get(&s.cand_lb, slots * (nl + 1));
  get(&s.cand_count, slots);
  get(&s.unit_prefix, slots * (nl + 2));
  get(&s.row_prefix, slots * (nl + 2));
  get(&s.group_q, slots * ix->L);
  get(&s.group_row, slots);
  get(&s.bound, slots);
  get(&s.kslots, slots * hg::kMaxK);
  get(&s.parts, slots * s.nparts * hg::kWarpListCap);
  get(&s.part_count, slots * s.nparts);
  get(&s.topk, slots * hg::kMaxK);
  get(&s.topk_count, slots);
  get(&s.sax_tab, slots * HG_PAA_SEGMENTS * HG_SAX_CARD);
  if (nl > (size_t)hg::kMaxLeavesSort) get(&s.sort_keys, slots * 4 * nl);
  get(&s.stats, 9);
  s.err = reinterpret_cast<int*>(s.stats + 8);
  get(&s.actl, 4);
  if (e == cudaSuccess) s.slots = (int)slots;
  return e;
}

// Scratch for groups of `want` queries, with a list of rows each if `lists`;
// where the device has no room for so many, for half as many, down to one (the
// caller reads group_room).  PSCAN, the epsilon and the nprobes search read no
// lists, which are most of the scratch of a large collection.
static hg_status ensure_scratch(hg_index* ix, uint32_t want, bool lists) {
  hg::QueryScratch& s = ix->s;
  if (s.slots == 0 || want > s.asked) {
    free_scratch(ix);
    for (uint32_t slots = want;; slots = std::max<uint32_t>(1, slots / 2)) {
      const cudaError_t e = alloc_scratch(ix, slots);
      if (e == cudaSuccess) break;
      free_scratch(ix);
      if (e != cudaErrorMemoryAllocation || slots == 1) return cuda_fail(e, "query scratch");
      cudaGetLastError();  // the failed allocation
    }
    s.asked = want;  // a smaller group was all there was room for: not tried again on each call
  }
  if (!lists || (s.list_slots > 0 && want <= s.list_asked)) return HG_OK;
  free_lists(ix);
  for (uint32_t slots = std::min<uint32_t>(want, (uint32_t)s.slots);; slots = std::max<uint32_t>(1, slots / 2)) {
    const cudaError_t e = dalloc(&s.list, (size_t)slots * ix->n);
    if (e == cudaSuccess) {
      s.list_slots = (int)slots;
      break;
    }
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "query scratch");
    cudaGetLastError();
    if (slots > 1) continue;
    // not one list beside this group's other scratch: a query at a time
    if (s.slots == 1) return cuda_fail(e, "query scratch");
    const uint32_t asked = s.asked;
    free_scratch(ix);
    const cudaError_t e1 = alloc_scratch(ix, 1);
    if (e1 != cudaSuccess) {
      free_scratch(ix);
      return cuda_fail(e1, "query scratch");
    }
    s.asked = asked;
  }
  s.list_asked = want;
  return HG_OK;
}

// queries per group, at most, of what ensure_scratch could get
static uint32_t group_room(const hg_index* ix, bool lists) {
  return (uint32_t)(lists ? std::min(ix->s.slots, ix->s.list_slots) : ix->s.slots);
}

static hg::Tree index_tree(const hg_index* ix) { return hg::Tree{ix->d.nodes, ix->d.root}; }

using ProfEvents = std::vector<std::pair<cudaEvent_t, cudaEvent_t>>;

struct Prof {
  ProfEvents ed, filter;
};

static hg_status timed_begin(ProfEvents* p, cudaStream_t st) {
  if (!p) return HG_OK;
  std::pair<cudaEvent_t, cudaEvent_t> ev;
  CK(cudaEventCreate(&ev.first));
  CK(cudaEventCreate(&ev.second));
  p->push_back(ev);
  CK(cudaEventRecord(ev.first, st));
  return HG_OK;
}

static hg_status timed_end(ProfEvents* p, cudaStream_t st) {
  if (p) CK(cudaEventRecord(p->back().second, st));
  return HG_OK;
}

static double drain(ProfEvents& p) {
  double ms = 0;
  for (auto& ev : p) {
    float t = 0;
    cudaEventElapsedTime(&t, ev.first, ev.second);
    ms += t;
    cudaEventDestroy(ev.first);
    cudaEventDestroy(ev.second);
  }
  p.clear();
  return ms;
}

static hg::EdArgs scan_args(hg_index* ix, const float* d_q, int k) {
  hg::QueryScratch& s = ix->s;
  hg::EdArgs e{};
  e.rows = ix->d.rows;
  e.ids = ix->d.ids;
  e.L = (int)ix->L;
  e.list_stride = ix->n;
  e.leaf_start = ix->d.leaf_start;
  e.leaf_size = ix->d.leaf_size;
  e.min_batch = 1;
  e.q = d_q;
  e.k = k;
  e.bound = s.bound;
  e.kslots = s.kslots;
  e.parts = s.parts;
  e.part_count = s.part_count;
  e.parts_stride = (uint32_t)s.nparts;
  e.stats = s.stats;
  return e;
}

static hg::MergeArgs merge_args(hg_index* ix, int nparts, int k, float* d_dist = nullptr, int64_t* d_id = nullptr) {
  hg::QueryScratch& s = ix->s;
  hg::MergeArgs m{};
  m.parts = s.parts;
  m.part_count = s.part_count;
  m.parts_stride = (uint32_t)s.nparts;
  m.nparts = nparts;
  m.k = k;
  m.topk = s.topk;
  m.topk_count = s.topk_count;
  m.bound = s.bound;
  m.dist_out = d_dist;
  m.id_out = d_id;
  return m;
}

static hg::PrepArgs prep_args(hg_index* ix, const float* d_q) {
  hg::QueryScratch& s = ix->s;
  hg::PrepArgs p{};
  p.q = d_q;
  p.L = (int)ix->L;
  p.tree = index_tree(ix);
  p.nleaves = (int)ix->leaves.size();
  p.seg_off = ix->d.leaf_seg_off;
  p.points = ix->d.leaf_points;
  p.sk = ix->d.leaf_sk;
  p.bp = ix->d.bp;
  p.approx_leaf = s.approx_leaf;
  p.bound = s.bound;
  p.kslots = s.kslots;
  p.topk_count = s.topk_count;
  p.counters = s.counters;
  return p;
}

// A group of queries (at most s.slots, consecutive at d_q) through the plain
// path, each launch serving all of them:
//   route, LB_EAPCA of every leaf, LB_SAX terms -> exact distances of the
//   approximate leaf -> merge: k-th bound, candidate leaves sorted by LB ->
//   LB_SAX filter -> exact distances of the survivors -> merge: answers.
static hg_status knn_group(hg_index* ix, const float* d_q, int slots, int k, const hg_knn_opts& o, float* d_dist,
                           int64_t* d_id, cudaStream_t st, Prof* prof, uint64_t* launches, bool has_floor = false,
                           float floor = 0.0f, const uint32_t* out_row = nullptr, uint32_t out_stride = 0) {
  hg::QueryScratch& s = ix->s;
  hg::DeviceIndex& d = ix->d;
  const int sms = hg::sm_count(ix->device);
  const int ed_blocks = sms * hg::ed_blocks_per_sm((int)ix->L);
  hg::EdArgs e = scan_args(ix, d_q, k);
  e.has_floor = has_floor ? 1 : 0;
  e.floor = floor;
  auto scan = [&](int blocks) -> hg_status {
    HCK(timed_begin(prof ? &prof->ed : nullptr, st));
    CK(hg::launch_ed_stream(e, slots, blocks, st));
    return timed_end(prof ? &prof->ed : nullptr, st);
  };
  if (o.mode == HG_MODE_PSCAN) {
    // every query's blocks resident at once: they walk the rows from the
    // front at the same pace, so the group reads most rows from L2
    const int blocks = std::max(1, ed_blocks / slots);
    CK(hg::launch_pscan_prep(s.bound, s.kslots, s.topk_count, slots, st));
    e.ident_count = ix->n;
    HCK(scan(blocks));
    CK(hg::launch_merge(merge_args(ix, blocks, k, d_dist, d_id), slots, st));
    *launches += 3;
    return HG_OK;
  }
  hg::PrepArgs p = prep_args(ix, d_q);
  p.lb = s.lb;
  p.sax_tab = o.use_lb_sax ? s.sax_tab : nullptr;
  CK(hg::launch_query_prep(p, slots, st));
  // the approximate leaf, with an unbounded k-th distance at the start: two
  // blocks per SM, as more warps would finish more rows of this leaf before
  // it tightens, and fewer leave HBM idle
  const int a_blocks =
      std::max(1, std::min(ed_blocks, o.approx_blocks > 0 ? o.approx_blocks : (int)ix->tune.approx_blocks_per_sm * sms));
  // a warp's entries: one row per slot of its lanes for a query alone; a
  // group keeps the GPU full by itself, so its warps take longer runs and
  // fewer blocks stage a query and sort a list.  Long rows: by the rows the
  // group's approximate leaves may hold against the GPU's 32 warps per SM
  // (12 queries, leaf 1,562, L = 16384: 0.93 ms at 4 entries, 1.20 at 8; 20
  // queries, leaf 2,000, L = 4096: 0.74 at 4, 0.67 at 8)
  const uint64_t warps = 32ull * sms;
  if (ix->L >= 4096) {
    const uint64_t rows = (uint64_t)slots * std::min<uint64_t>(ix->leaf_size, ix->n);
    e.few_rows = slots == 1 && 2 * rows <= warps ? UINT32_MAX : 0;
    e.min_batch = slots > 1 && rows >= 6 * warps ? 8u : 4u;
  } else {
    e.min_batch = slots > 1 ? 32u : 8u;
  }
  e.ident_leaf = s.approx_leaf;
  HCK(scan(a_blocks));
  hg::SelectArgs sel{};
  sel.lb = s.lb;
  sel.nleaves = (int)ix->leaves.size();
  sel.approx_leaf = s.approx_leaf;
  sel.leaf_start = d.leaf_start;
  sel.leaf_size = d.leaf_size;
  sel.cand = s.cand;
  sel.cand_lb = s.cand_lb;
  sel.cand_count = s.cand_count;
  sel.unit_prefix = s.unit_prefix;
  // The bound after the approximate leaf is close to the last one (seeding with
  // the next eight leaves drops 2% of the chunks read), so the leaves' order
  // matters less than where their rows lie: in file order the queries of a
  // group meet each other's rows in L2, and nothing is sorted.  16 queries of
  // 8M x 256 4.78 -> 4.53 ms, 32 of 2M x 128 (leaf 500, LB_SAX) 1.45 -> 1.31,
  // one of 1M x 256 (leaf 1,000) 148 -> 136 us.  In LB order: an unbounded
  // search, the seeded one, which takes the first of them alone, and long
  // series, whose few rows still lower the bound (12 of 100k x 16384 3.73 ms,
  // 3.88 in file order).
  sel.by_file = ix->L < 4096 && o.approx_leaves <= 1;
  sel.row_prefix = o.use_lb_sax ? nullptr : s.row_prefix;
  sel.gkeys = s.sort_keys;
  CK(hg::launch_merge_select(merge_args(ix, a_blocks, k), sel, slots, st));
  hg::FilterArgs f{};
  f.sax = d.sax;
  f.L = e.L;
  f.nleaves = sel.nleaves;
  f.leaf_start = d.leaf_start;
  f.leaf_size = d.leaf_size;
  f.cand = s.cand;
  f.cand_lb = s.cand_lb;
  f.cand_count = s.cand_count;
  f.unit_prefix = s.unit_prefix;
  f.row_prefix = s.row_prefix;
  f.sax_tab = s.sax_tab;
  f.bound = s.bound;
  f.list = s.list;
  f.list_stride = ix->n;
  f.stats = s.stats;
  f.err = s.err;
  e.ident_leaf = nullptr;
  e.list = s.list;
  // the rows left for one query over long series: a warp each while there are
  // warps for all, 8 lanes above.  LB_SAX often leaves a thousand rows; without
  // it, or for a query unlike any row, most of the collection is left, and only
  // the device knows.  One query of 100k x 16384, leaf 1,562, whole calls: a warp
  // per row whatever the count / 8 lanes / by the count: 30k rows 0.84 / 0.61 /
  // 0.61 ms, white noise (99k rows) 2.22 / 1.36 / 1.36, 1,500 rows 0.341 / 0.407 /
  // 0.345.  The launch that returns at once takes 4 us.
  e.few_rows = ix->L >= 4096 && slots == 1 ? (uint32_t)warps : 0;
  // one LB_SAX filter block is resident per SM (eight that only list rows): a
  // query alone takes them all, a group a share each, with some to spare for
  // its larger queries
  const int f_blocks = std::min(sms, std::max(1, 4 * sms / slots)) * (o.use_lb_sax ? 1 : 8);
  auto filter_scan_merge = [&](uint32_t* count, float* dist, int64_t* id) -> hg_status {
    f.list_count = count;
    HCK(timed_begin(prof ? &prof->filter : nullptr, st));
    CK(o.use_lb_sax ? hg::launch_lbsax_filter(f, slots, f_blocks, st) : hg::launch_list_rows(f, slots, f_blocks, st));
    HCK(timed_end(prof ? &prof->filter : nullptr, st));
    e.list_count = count;
    HCK(scan(ed_blocks));
    // the merge folds the earlier stages' top-k into the result
    hg::MergeArgs m = merge_args(ix, ed_blocks, k, dist, id);
    m.out_row = out_row;
    m.out_stride = out_stride;
    CK(hg::launch_merge(m, slots, st));
    *launches += e.few_rows ? 4 : 3;
    return HG_OK;
  };
  // greedy seeding (the paper's L_max): the next approx_leaves - 1
  // candidates in LB order, scanned before the rest so that the bound the
  // rest is filtered against is tighter
  const int seed = (o.mode == HG_MODE_PLAIN && o.approx_leaves > 1) ? o.approx_leaves - 1 : 0;
  if (seed > 0) {
    f.cand_hi = seed;
    HCK(filter_scan_merge(s.counters + 4, nullptr, nullptr));
    f.cand_lo = seed;
    f.cand_hi = 0;
  }
  HCK(filter_scan_merge(s.counters + 2, d_dist, d_id));
  *launches += 3;
  return HG_OK;
}

static hg_status knn_batch_impl(hg_index* ix, const float* d_Q, uint32_t nq, const uint32_t* ks, uint32_t kmax,
                                const hg_knn_opts& o, float* d_dist, int64_t* d_id, cudaStream_t st,
                                hg_query_stats* stats, bool host_io = false);

// Best-first queue of the approximate searches: a binary min-heap on the
// node lower bound that moves an entry past another only when strictly
// smaller and, between equal children, takes the left one -- the order in
// which the reference's pqueue (pqueue.c, cmp_pri in hercules_query_engine.h)
// pops equal bounds, so both visit nodes in the same sequence.
struct PqEntry {
  float d;
  int node;
};
static void pq_push(std::vector<PqEntry>& h, PqEntry e) {
  h.push_back(e);
  size_t i = h.size() - 1;
  while (i > 0) {
    const size_t p = (i - 1) / 2;
    if (!(h[p].d > h[i].d)) break;
    std::swap(h[p], h[i]);
    i = p;
  }
}
static bool pq_pop(std::vector<PqEntry>& h, PqEntry* out) {
  if (h.empty()) return false;
  *out = h[0];
  h[0] = h.back();
  h.pop_back();
  size_t i = 0;
  for (;;) {
    const size_t l = 2 * i + 1, r = l + 1;
    if (l >= h.size()) break;
    const size_t c = (r < h.size() && h[l].d > h[r].d) ? r : l;
    if (!(h[i].d > h[c].d)) break;
    std::swap(h[i], h[c]);
    i = c;
  }
  return true;
}

// epsilon-approximate search (exact_de_knn_search with epsilon,
// hercules_query_engine.c:2215-2448) or nprobes search (exact_ng_knn_search,
// :2623-2796) of one query.  The tree walk runs on the host with the
// reference's LB_EAPCA arithmetic on the tree's own envelopes (internal
// nodes included, as the reference prunes with them); every leaf scan is a
// distance-stream launch over the leaf's rows followed by the merge into the
// query's top-k on the device.
//  - epsilon: the walk collects leaves with the k-th distance of the
//    approximate leaf (pop stops at LB > kth/(1+eps), children pushed at
//    LB < kth/(1+eps)); the leaves are then taken in file_pos order, each
//    scanned only if LB <= kth/(1+eps) with the k-th distance the reference
//    holds at that moment: the value read before the last row of the
//    previously scanned leaf.  So each leaf is scanned as its rows but the
//    last, then the last row, and the k-th distance between the two is kept
//    for the next leaf's test (k_leaf_gate, k_stale_copy; no host wait).
//  - nprobes: a leaf is scanned when popped, at most nprobes leaves with the
//    approximate one; the walk stops at a node whose LB exceeds the
//    approximate leaf's best distance; children are pushed at LB < the
//    current k-th distance (read back after each leaf).
static hg_status knn_approx_one(hg_index* ix, const float* d_q, int k, const hg_knn_opts& o, float* d_dist,
                                int64_t* d_id, cudaStream_t st) {
  hg::QueryScratch& s = ix->s;
  const int L = (int)ix->L;
  const int sms = hg::sm_count(ix->device);
  const int ed_blocks = sms * hg::ed_blocks_per_sm(L);
  hg::EdArgs e = scan_args(ix, d_q, k);
  CK(hg::launch_query_prep(prep_args(ix, d_q), 1, st));
  e.ident_leaf = s.approx_leaf;
  CK(hg::launch_ed_stream(e, 1, ed_blocks, st));
  CK(hg::launch_merge(merge_args(ix, ed_blocks, k), 1, st));
  std::vector<float> q(L);
  int approx = -1, cnt = 0;
  uint32_t bound_bits = 0;
  unsigned long long best_key = ~0ull;
  CK(cudaMemcpyAsync(q.data(), d_q, sizeof(float) * L, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&approx, s.approx_leaf, sizeof approx, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&cnt, s.topk_count, sizeof cnt, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&bound_bits, s.bound, sizeof bound_bits, cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&best_key, s.topk, sizeof best_key, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  // the reference's k-th distance: FLT_MAX until k results are held
  auto kth_of = [&](int c, uint32_t bits) {
    float f;
    memcpy(&f, &bits, sizeof f);
    return c >= k ? f : FLT_MAX;
  };
  float kth = kth_of(cnt, bound_bits);
  float best = FLT_MAX;
  if (cnt > 0) {
    const uint32_t hi = (uint32_t)(best_key >> 32);
    memcpy(&best, &hi, sizeof best);
  }
  // knn_results[0].node: the approximate leaf once it produced a result
  const int approx_node = (cnt > 0 && approx >= 0) ? ix->leaves[approx] : -1;
  auto lb_of = [&](int node) {
    const hg::Node& n = ix->nodes[node];
    return hg_lb_eapca(q.data(), (int)n.points.size(), n.points.data(), n.sk.data());
  };
  int* flag = reinterpret_cast<int*>(s.actl + 1);
  uint32_t* stale = s.actl + 0;
  // one leaf: its rows but the last, the stale k-th distance, the last row
  auto scan_leaf = [&](int node, float lb, float eps1) -> hg_status {
    const hg::Node& n = ix->nodes[node];
    if (n.node_size == 0) return HG_OK;
    CK(hg::launch_leaf_gate(lb, eps1, stale, flag, s.stats + 3, st));
    e.gate = flag;
    e.ident_leaf = nullptr;
    const uint64_t first = n.file_pos, count = n.node_size;
    if (count > 1) {
      e.ident_first = first;
      e.ident_count = count - 1;
      CK(hg::launch_ed_stream(e, 1, ed_blocks, st));
      CK(hg::launch_merge(merge_args(ix, ed_blocks, k), 1, st));
    }
    CK(hg::launch_stale_copy(flag, s.bound, stale, st));
    e.ident_first = first + count - 1;
    e.ident_count = 1;
    CK(hg::launch_ed_stream(e, 1, 1, st));
    CK(hg::launch_merge(merge_args(ix, 1, k), 1, st));
    return HG_OK;
  };
  std::vector<PqEntry> pq;
  pq_push(pq, PqEntry{lb_of(0), 0});  // nodes[0] is the root
  PqEntry it;
  if (o.nprobes > 0) {
    int probes = 1;
    const float never = -FLT_MAX;  // a popped leaf is always scanned
    while (pq_pop(pq, &it) && probes < o.nprobes) {
      if (it.d > best) break;
      const hg::Node& n = ix->nodes[it.node];
      if (n.is_leaf) {
        HCK(scan_leaf(it.node, never, 1.0f));
        ++probes;
        CK(cudaMemcpyAsync(&cnt, s.topk_count, sizeof cnt, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&bound_bits, s.bound, sizeof bound_bits, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        kth = kth_of(cnt, bound_bits);
      } else {
        for (int c : {n.left, n.right}) {
          const float lb = lb_of(c);
          if (lb < kth && c != approx_node) pq_push(pq, PqEntry{lb, c});
        }
      }
    }
  } else {
    const float eps1 = 1.0f + o.epsilon;
    std::vector<PqEntry> cand;
    while (pq_pop(pq, &it)) {
      if (it.d > kth / eps1) break;
      const hg::Node& n = ix->nodes[it.node];
      if (n.is_leaf) {
        cand.push_back(it);
      } else {
        for (int c : {n.left, n.right}) {
          const float lb = lb_of(c);
          if (lb < kth / eps1 && c != approx_node) pq_push(pq, PqEntry{lb, c});
        }
      }
    }
    std::stable_sort(cand.begin(), cand.end(), [&](const PqEntry& a, const PqEntry& b) {
      return ix->nodes[a.node].file_pos < ix->nodes[b.node].file_pos;
    });
    uint32_t kth_bits;
    memcpy(&kth_bits, &kth, sizeof kth_bits);
    CK(cudaMemcpyAsync(stale, &kth_bits, sizeof kth_bits, cudaMemcpyHostToDevice, st));
    for (const PqEntry& c : cand) HCK(scan_leaf(c.node, c.d, eps1));
  }
  CK(hg::launch_emit(s.topk, s.topk_count, k, d_dist, d_id, st));
  CK(cudaStreamSynchronize(st));  // kth_bits and the host vectors leave scope
  return HG_OK;
}

// k above kMaxK: rounds of at most kMaxK answers.  Round r returns the next
// smallest distinct distances strictly above the last distance of round
// r - 1 (the distance stream admits only rows above that floor; pruning by
// LB_EAPCA / LB_SAX against the round's own k-th bound is unchanged), so
// the rounds together are the k smallest distinct distances, each with its
// lowest id -- the answer of one search with that k.  A round that comes
// back short means the collection has no more distances: the remaining
// entries are +inf / -1.  The host reads each round's last distance back.
static hg_status knn_rounds(hg_index* ix, const float* d_q, uint32_t k, const hg_knn_opts& o, float* d_dist,
                            int64_t* d_id, cudaStream_t st, Prof* prof, uint64_t* launches) {
  hg::QueryScratch& s = ix->s;
  uint32_t done = 0;
  bool has_floor = false;
  float floor = 0.0f;
  while (done < k) {
    const int kr = (int)std::min<uint32_t>((uint32_t)hg::kMaxK, k - done);
    HCK(knn_group(ix, d_q, 1, kr, o, d_dist ? d_dist + done : nullptr, d_id ? d_id + done : nullptr, st, prof, launches,
                  has_floor, floor));
    int cnt = 0;
    unsigned long long last = 0;
    CK(cudaMemcpyAsync(&cnt, s.topk_count, sizeof cnt, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&last, s.topk + (kr - 1), sizeof last, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    done += (uint32_t)kr;
    if (cnt < kr) {
      if (done < k) {
        // nothing above this round's distances: the rest is empty
        CK(cudaMemsetAsync(s.topk_count, 0, sizeof(int), st));
        CK(hg::launch_emit(s.topk, s.topk_count, (int)(k - done), d_dist ? d_dist + done : nullptr,
                           d_id ? d_id + done : nullptr, st));
        ++*launches;
      }
      break;
    }
    has_floor = true;
    const uint32_t bits = (uint32_t)(last >> 32);
    memcpy(&floor, &bits, sizeof floor);
  }
  return HG_OK;
}

constexpr size_t kHostIoKeep = 64u << 20;

template <class T>
static hg_status grow_io(T** p, size_t* cap, size_t bytes) {
  if (*cap >= bytes && *p) return HG_OK;
  dfree(*p);
  *cap = 0;
  unsigned char* b = nullptr;
  CK(dalloc(&b, bytes));
  *p = reinterpret_cast<T*>(b);
  *cap = bytes;
  return HG_OK;
}

// frees the copies that are larger than `keep`
static void trim_io(hg::HostIo& io, size_t keep) {
  if (io.q_cap > keep) {
    dfree(io.q);
    io.q_cap = 0;
  }
  if (io.out_cap > keep) {
    dfree(io.out);
    io.out_cap = 0;
  }
}

// host_out: if set, host_bytes from device memory host_src (the answers) are
// copied there with the call's counters, before its one synchronisation.
static hg_status knn_device_impl(hg_index* ix, const float* d_queries, uint32_t nq, uint32_t k,
                                 const hg_knn_opts* opts, float* d_dist, int64_t* d_id, cudaStream_t st,
                                 hg_query_stats* stats, void* host_out = nullptr, const void* host_src = nullptr,
                                 size_t host_bytes = 0) {
  if (!ix || (!d_queries && nq)) return set_error(HG_ERR_ARG, "hg_knn: null argument");
  if (k == 0) return set_error(HG_ERR_ARG, "hg_knn: k must be positive");
  if (ix->L > 16384) return set_error(HG_ERR_LIMIT, "hg_knn: series longer than 16384");
  hg_knn_opts o{};
  if (opts) o = *opts;
  if (o.mode == HG_MODE_BATCH) return knn_batch_impl(ix, d_queries, nq, nullptr, k, o, d_dist, d_id, st, stats);
  const bool approx = o.mode == HG_MODE_PLAIN && (o.epsilon > 0.0f || o.nprobes > 0);
  if (o.epsilon < 0.0f || o.nprobes < 0 || !(o.epsilon == o.epsilon))
    return set_error(HG_ERR_ARG, "hg_knn: epsilon and nprobes must not be negative");
  // k above kMaxK is answered in rounds (exact); the approximate searches
  // depend on the k-th distance at every step, so they keep the limit
  if (approx && (int)k > hg::kMaxK)
    return set_error(HG_ERR_LIMIT, "hg_knn: k above 224 with epsilon or nprobes");
  CK(cudaSetDevice(ix->device));
  // rounds and approximate searches follow one query at a time
  const bool grouped = !approx && (int)k <= hg::kMaxK, lists = !approx && o.mode != HG_MODE_PSCAN;
  const uint32_t want = grouped ? group_slots(ix, nq) : 1;
  HCK(ensure_scratch(ix, want, lists));
  if (!st) st = ix->stream;
  for (cudaEvent_t& e : ix->ev)
    if (!e) CK(cudaEventCreate(&e));
  CK(cudaMemsetAsync(ix->s.stats, 0, sizeof(unsigned long long) * 9, st));
  Prof prof;
  CK(cudaEventRecord(ix->ev[0], st));
  uint64_t launches = 0;
  const uint32_t per = std::min(want, group_room(ix, lists));
  for (uint32_t i = 0; i < nq; i += per) {
    const float* qi = d_queries + (uint64_t)i * ix->L;
    float* di = d_dist ? d_dist + (uint64_t)i * k : nullptr;
    int64_t* ii = d_id ? d_id + (uint64_t)i * k : nullptr;
    Prof* pr = o.profile ? &prof : nullptr;
    if (approx) HCK(knn_approx_one(ix, qi, (int)k, o, di, ii, st));
    else if (grouped) HCK(knn_group(ix, qi, (int)std::min(per, nq - i), (int)k, o, di, ii, st, pr, &launches));
    else HCK(knn_rounds(ix, qi, k, o, di, ii, st, pr, &launches));
  }
  CK(cudaEventRecord(ix->ev[1], st));
  unsigned long long hs[9];  // counters, error flag
  CK(cudaMemcpyAsync(hs, ix->s.stats, sizeof hs, cudaMemcpyDeviceToHost, st));
  if (host_out) CK(cudaMemcpyAsync(host_out, host_src, host_bytes, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  const int ferr = (int)(uint32_t)hs[8];
  float ms = 0;
  if (stats) cudaEventElapsedTime(&ms, ix->ev[0], ix->ev[1]);
  if (ferr) return set_error(HG_ERR_TIMEOUT, "hg_knn: an LB_SAX filter wait timed out");
  const size_t ed_launches = prof.ed.size(), filter_launches = prof.filter.size();
  const double scan_ms = drain(prof.ed);
  const double filter_ms = drain(prof.filter);
  if (stats) {
    memset(stats, 0, sizeof *stats);
    stats->queries = nq;
    stats->rows_considered = hs[0];
    stats->chunks_loaded = hs[1];
    stats->rows_lbsax_pruned = hs[2];
    stats->leaves_scanned = hs[3];
    stats->rows_completed = hs[4];
    stats->rows_visited = hs[5];
    stats->device_ms = ms;
    stats->scan_launches = ed_launches;
    stats->scan_ms = scan_ms;
    stats->filter_launches = filter_launches;
    stats->filter_ms = filter_ms;
    stats->kernel_launches = launches;
  }
  return HG_OK;
}


// ---------------------------------------------------------------------------
// batched queries: BF16 tensor-core filter + exact re-rank (hg_batch.cu)
// ---------------------------------------------------------------------------

constexpr uint32_t kDefaultBucket = 65536;
constexpr int kBatchRetries = 3;  // filter rounds after the first for overflowed buckets

// TMA descriptor of a row-major n x L BF16 matrix, boxes of 64 columns
// (128 bytes, the swizzle span) x box_rows rows, 128-byte swizzle, zero fill
// outside the matrix.  The encoder comes from the driver through the runtime.
static hg_status encode_bf16_map(CUtensorMap* map, const void* base, uint64_t n, uint32_t L, uint32_t box_rows) {
  // the driver's entry point is process-wide; a function-local static is
  // initialised once even when several threads get here first
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  if (!encode) return set_error(HG_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (n == 0 || n >= (1ull << 31) || (L * 2) % 16 != 0)
    return set_error(HG_ERR_LIMIT, "BF16 tensor map: n must be below 2^31 and L a multiple of 8");
  const cuuint64_t dims[2] = {L, n};
  const cuuint64_t strides[1] = {(cuuint64_t)L * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_error(HG_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return HG_OK;
}

static hg_status encode_query_maps(hg::QueryMaps* m, const void* base, uint64_t n, uint32_t L) {
  HCK(encode_bf16_map(&m->q256, base, n, L, hg::kBatchQueryTile));
  HCK(encode_bf16_map(&m->q128, base, n, L, hg::kBatchQueryTile / 2));
  return encode_bf16_map(&m->q64, base, n, L, hg::kBatchBoundQueries);
}

static hg_status make_batch_data(hg_index* ix, cudaStream_t st, uint16_t** x) {
  hg::BatchData& b = ix->bd;
  const uint64_t nt = (ix->n + hg::kBatchTileRows - 1) / hg::kBatchTileRows;
  CK(dalloc(x, ix->n * ix->L));
  CK(dalloc(&b.xmeta, ix->n));
  CK(dalloc(&b.tile_meta, nt));
  CK(hg::launch_rows_to_bf16(ix->d.rows, nullptr, ix->n, (int)ix->L, *x, b.xmeta, st));
  CK(hg::launch_tile_norms(b.xmeta, ix->n, b.tile_meta, st));
  return encode_bf16_map(&b.rows_map, *x, ix->n, ix->L, 128);
}

// b.xbf says that all of it is there
static hg_status ensure_batch_data(hg_index* ix, cudaStream_t st) {
  hg::BatchData& b = ix->bd;
  if (b.xbf) return HG_OK;
  uint16_t* x = nullptr;
  const hg_status s = make_batch_data(ix, st, &x);
  if (s == HG_OK) {
    b.xbf = x;
    return HG_OK;
  }
  dfree(x);
  dfree(b.xmeta);
  dfree(b.tile_meta);
  return s;
}

static hg_status ensure_batch_scratch(hg_index* ix, uint32_t nq, uint32_t bucket_cap, uint32_t bm_cap,
                                      uint32_t nitems, uint32_t kmax) {
  hg::BatchScratch& b = ix->bs;
  if (nq > b.nq_cap) {
    dfree(b.qlist);
    dfree(b.seg_rows);
    dfree(b.seg_prefix);
    dfree(b.qbound);
    dfree(b.parts);
    dfree(b.part_cnt);
    dfree(b.qbf);
    dfree(b.qmeta);
    dfree(b.qperm);
    dfree(b.approx);
    dfree(b.kq);
    dfree(b.slots);
    dfree(b.bound);
    dfree(b.init);
    dfree(b.init_cnt);
    dfree(b.bucket_cnt);
    dfree(b.ok);
    // sized for nq_cap queries too, allocated by the caller
    dfree(b.qlist2);
    dfree(b.qin);
    dfree(b.out_dist);
    dfree(b.out_id);
    uint16_t* q = nullptr;
    CK(dalloc(&q, (size_t)nq * ix->L));
    b.qbf = q;
    CK(dalloc(&b.qmeta, nq));
    CK(dalloc(&b.qperm, nq));
    CK(dalloc(&b.approx, nq));
    CK(dalloc(&b.kq, nq));
    CK(dalloc(&b.slots, nq));
    CK(dalloc(&b.bound, nq));
    CK(dalloc(&b.init, (size_t)nq * hg::kMaxK));
    CK(dalloc(&b.init_cnt, nq));
    CK(dalloc(&b.bucket_cnt, nq));
    CK(dalloc(&b.ok, nq));
    CK(dalloc(&b.qlist, nq));
    CK(dalloc(&b.seg_rows, nq));
    CK(dalloc(&b.seg_prefix, (size_t)nq + 1));
    CK(dalloc(&b.qbound, nq));
    CK(dalloc(&b.part_cnt, (size_t)nq + hg::kBatchSegTarget));
    b.nq_cap = nq;
    ++b.gen;  // a captured pipeline holds the old addresses
    b.bucket_cap = 0;
    b.bm_cap = 0;
    b.parts_kmax = 0;
  }
  // survivor pairs: room for 16,384 per query of the batch and a block begun
  // by every filter warp, at most 2^28
  const uint64_t begun = (uint64_t)hg::sm_count(ix->device) * hg::kBatchPairWarps * hg::kBatchPairBlock;
  const uint32_t pairs_cap = (uint32_t)std::min<uint64_t>((uint64_t)b.nq_cap * 16384 + begun, 1ull << 28);
  if (pairs_cap > b.pairs_cap || !b.pairs) {
    dfree(b.pairs);
    CK(dalloc(&b.pairs, pairs_cap));
    b.pairs_cap = pairs_cap;
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  if (kmax > b.parts_kmax || !b.parts) {
    dfree(b.parts);
    CK(dalloc(&b.parts, ((size_t)b.nq_cap + hg::kBatchSegTarget) * kmax));
    b.parts_kmax = kmax;
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  if (!b.ctl) {
    CK(dalloc(&b.ctl, 1));
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  if ((uint64_t)b.nq_cap * bucket_cap > (uint64_t)b.nq_cap * b.bucket_cap || !b.bucket) {
    dfree(b.bucket);
    CK(dalloc(&b.bucket, (size_t)b.nq_cap * bucket_cap));
    b.bucket_cap = bucket_cap;
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  if (bm_cap > b.bm_cap || !b.bm) {
    dfree(b.bm);
    CK(dalloc(&b.bm, (size_t)b.nq_cap * bm_cap));
    b.bm_cap = bm_cap;
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  if (nitems > b.items_cap || !b.items) {
    dfree(b.items);
    CK(dalloc(&b.items, std::max<uint32_t>(nitems, 1)));
    b.items_cap = std::max<uint32_t>(nitems, 1);
    ++b.gen;  // a captured pipeline holds the old addresses
  }
  return HG_OK;
}

// Buffers of the pruned filter for b.nq_cap queries; *ok = false when they
// would not fit their limits (the batch then filters every row): the kept
// (leaf, query) lists within 1 GiB, the query panel within a quarter of the
// free device memory (1 to 16 GiB) or one copy of the batch, whichever is
// larger.
static hg_status ensure_prune_scratch(hg_index* ix, bool* ok) {
  hg::BatchScratch& b = ix->bs;
  const uint64_t nl = ix->leaves.size(), nq = b.nq_cap, L = ix->L;
  *ok = nl > 0 && nl * nq * 4 <= (1ull << 30);
  if (!*ok) return HG_OK;
  if (!b.seg_uid) {
    // distinct (start, end) segments over the leaves, in leaf_points order
    std::map<std::pair<int, int>, int> ids;
    std::vector<short> us, ue;
    std::vector<int> uid;
    for (int l : ix->leaves) {
      int start = 0;
      for (short e : ix->nodes[l].points) {
        auto it = ids.emplace(std::make_pair(start, (int)e), (int)us.size());
        if (it.second) {
          us.push_back((short)start);
          ue.push_back(e);
        }
        uid.push_back(it.first->second);
        start = e;
      }
    }
    b.nu = (int)us.size();
    CK(dalloc(&b.useg_start, std::max<size_t>(us.size(), 1)));
    CK(dalloc(&b.useg_end, std::max<size_t>(ue.size(), 1)));
    CK(dalloc(&b.seg_uid, std::max<size_t>(uid.size(), 1)));
    if (!us.empty()) {
      CK(cudaMemcpy(b.useg_start, us.data(), sizeof(short) * us.size(), cudaMemcpyHostToDevice));
      CK(cudaMemcpy(b.useg_end, ue.data(), sizeof(short) * ue.size(), cudaMemcpyHostToDevice));
      CK(cudaMemcpy(b.seg_uid, uid.data(), sizeof(int) * uid.size(), cudaMemcpyHostToDevice));
    }
  }
  if ((uint64_t)b.nu * nq * sizeof(float2) > (1ull << 30)) {
    *ok = false;
    return HG_OK;
  }
  if (b.prune_nq >= nq && b.leaf_q) return HG_OK;
  dfree(b.leaf_cnt);
  dfree(b.leaf_q);
  dfree(b.leaf_poff);
  dfree(b.leaf_ioff);
  dfree(b.panel_list);
  dfree(b.panel_bf);
  dfree(b.items3);
  dfree(b.segstats);
  b.prune_nq = 0;
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  const uint64_t budget = std::min<uint64_t>(16ull << 30, std::max<uint64_t>(1ull << 30, free_b / 4));
  const uint64_t panel = std::min<uint64_t>(nl * nq, std::max<uint64_t>(nq, budget / (2 * L)));
  // items for the narrowest work item (8 tiles): chunks of every leaf x its query tiles
  const uint64_t ntiles = (ix->n + hg::kBatchTileRows - 1) / hg::kBatchTileRows;
  // and 2 kBatchItemTarget more where narrower ones even out a small batch: the
  // item list never overflows
  const uint64_t items =
      (ntiles / 8 + 2 * nl) * ((nq + hg::kBatchQueryTile - 1) / hg::kBatchQueryTile) + 2 * hg::kBatchItemTarget;
  if (panel >= (1ull << 32) || items >= (1ull << 31)) {
    *ok = false;
    return HG_OK;
  }
  CK(dalloc(&b.leaf_cnt, nl));
  CK(dalloc(&b.leaf_q, nl * nq));
  CK(dalloc(&b.leaf_poff, nl));
  CK(dalloc(&b.leaf_ioff, nl));
  CK(dalloc(&b.panel_list, panel));
  uint16_t* p = nullptr;
  CK(dalloc(&p, panel * L));
  b.panel_bf = p;
  CK(dalloc(&b.items3, items));
  CK(dalloc(&b.segstats, std::max<uint64_t>((uint64_t)b.nu * nq, 1)));
  b.panel_cap = (uint32_t)panel;
  b.items3_cap = (uint32_t)items;
  HCK(encode_query_maps(&b.panel_maps, b.panel_bf, panel, (uint32_t)L));
  b.prune_nq = (uint32_t)nq;
  ++b.gen;  // a captured pipeline holds the old addresses
  return HG_OK;
}

// Error-bound coefficients of the BF16 filter for series length L (see
// hg_batch.cu): c_acc = L 2^-20 (FP32 accumulation on the tensor cores) and
// c_sq = (L/8 + 16) 2^-22, both rounded up to float.
static void filter_coefficients(uint32_t L, float* c_acc, float* c_sq) {
  *c_acc = std::nextafter((float)(L * std::ldexp(1.0, -20)), INFINITY);
  *c_sq = std::nextafter((float)((L / 8.0 + 16.0) * std::ldexp(1.0, -22)), INFINITY);
}

// Bound-pass plan of every leaf for `want` candidate rows per query: slots
// per 128-row tile (enough for `want` where the leaf has the rows, at most
// kBatchMaxSlots per query) and the tiles used.
static hg_status ensure_leaf_plan(hg_index* ix, uint64_t want, cudaStream_t st) {
  hg::BatchScratch& b = ix->bs;
  const int nl = (int)ix->leaves.size();
  if (b.leaf_plan && b.plan_want == want) return HG_OK;
  const uint32_t T = hg::kBatchTileRows;
  auto sub_of = [&](uint32_t tiles) {
    uint32_t sub = 1;
    while (sub < 16 && (uint64_t)std::max<uint32_t>(tiles, 1) * sub < want) sub <<= 1;
    return sub;
  };
  std::vector<hg::LeafPlan> plan(nl);
  uint32_t bm_cap = 1;
  for (int l = 0; l < nl; ++l) {
    const Node& nd = ix->nodes[ix->leaves[l]];
    const uint32_t tiles = (uint32_t)((nd.node_size + T - 1) / T);
    plan[l].start = nd.file_pos;
    plan[l].size = nd.node_size;
    plan[l].sub = sub_of(tiles);
    plan[l].pad = 0;
    bm_cap = std::max<uint32_t>(bm_cap, (uint32_t)std::min<uint64_t>(hg::kBatchMaxSlots, (uint64_t)tiles * plan[l].sub));
  }
  uint32_t max_use = 0;
  for (int l = 0; l < nl; ++l) {
    const uint32_t tiles = (plan[l].size + T - 1) / T;
    plan[l].use_tiles = std::min<uint32_t>(tiles, bm_cap / plan[l].sub);
    max_use = std::max(max_use, plan[l].use_tiles);
  }
  if (!b.leaf_plan) {
    CK(dalloc(&b.leaf_plan, nl));
    if (nl > hg::kMaxLeavesSort) CK(dalloc(&b.group_cnt, 2 * (size_t)nl));
    CK(dalloc(&b.leaf_qoff, nl + 1));
    CK(dalloc(&b.leaf_qcnt, nl + 1));
    CK(dalloc(&b.item_off, nl + 1));
  }
  CK(cudaMemcpyAsync(b.leaf_plan, plan.data(), sizeof(hg::LeafPlan) * nl, cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));
  b.plan_want = want;
  b.plan_bm_cap = bm_cap;
  b.plan_max_use = max_use;
  ++b.gen;
  return HG_OK;
}

// One round of a batch, after the queries are in b.qin and their k in b.kq, as
// one stream-ordered sequence with no host decision inside (so it can be
// captured in a CUDA graph).  Round 0 routes and groups the queries on the
// device and runs the bound pass; every round filters, re-ranks and lists the
// queries left to retry.  A retry round is launched only when the one before
// left it queries: three empty rounds of twelve kernels each cost a small
// batch a third of its time (100k x 256, 64 queries: 300 -> 127 us on the device, with
// the stamps, counters and overflow marks folded into the kernels beside them).
static hg_status enqueue_round(hg_index* ix, int round, uint32_t nq, uint32_t kmax, uint32_t bucket_cap,
                               const hg::QueryMaps& qmaps, bool prune, cudaStream_t st, uint64_t* launches) {
  hg::BatchScratch& b = ix->bs;
  hg::BatchCtl* c = b.ctl;
  const hg::DeviceIndex& d = ix->d;
  const uint32_t L = ix->L;
  const int sms = hg::sm_count(ix->device);
  const int nl = (int)ix->leaves.size();
  uint64_t n_launch = 0;
  hg::BatchGemm g{};
  g.L = (int)L;
  g.nrows = ix->n;
  g.xmeta = ix->bd.xmeta;
  g.tile_meta = ix->bd.tile_meta;
  g.qmeta = b.qmeta;
  g.nq = (int)nq;
  g.bm = b.bm;
  g.bm_cap = b.plan_bm_cap;
  g.tiles_per_item = ix->tune.filter_tiles_per_item;
  filter_coefficients(L, &g.c_acc, &g.c_sq);
  g.bound = b.bound;
  g.pairs = b.pairs;
  g.pairs_cnt = c->heads + 1;
  g.pairs_cap = b.pairs_cap;
  g.err = reinterpret_cast<int*>(c->heads + 3);
  hg::BatchRank r{};
  r.rows = d.rows;
  r.ids = d.ids;
  r.Q = b.qin;
  r.L = (int)L;
  r.nq = (int)nq;
  r.kq = b.kq;
  r.kmax = (int)kmax;
  r.bm = b.bm;
  r.bm_cap = b.plan_bm_cap;
  r.slots_of_query = b.slots;
  r.bound = b.bound;
  r.init = b.init;
  r.init_cnt = b.init_cnt;
  r.bucket = b.bucket;
  r.bucket_cnt = b.bucket_cnt;
  r.bucket_cap = bucket_cap;
  r.pairs_cnt = c->heads + 1;
  r.pairs_cap = b.pairs_cap;
  r.dist_out = b.out_dist;
  r.id_out = b.out_id;
  r.ok_out = b.ok;
  r.stats = c->stats;
  r.seg_rows = b.seg_rows;
  r.seg_prefix = b.seg_prefix;
  r.qbound = b.qbound;
  r.parts = b.parts;
  r.part_cnt = b.part_cnt;
  r.heads = c->heads + 2;
  uint32_t* lists[2] = {b.qlist, b.qlist2};
  const uint32_t* list = round == 0 ? nullptr : lists[(round - 1) & 1];
  const uint32_t* n_dev = round == 0 ? nullptr : c->ctrl + 4 + round;
  r.qlist = list;
  r.nlist = (int)nq;
  r.nlist_dev = n_dev;
  // the narrowest work item: a resident query tile (L <= 256) is loaded once
  // per item, so an item has at least four row tiles; a streamed one is read
  // for every two row tiles whatever the item's length
  const uint32_t tpi_min = L <= 256 ? 4 : 2;
  uint32_t* pctl = round == 0 ? c->pctl : c->pctl + 8;
  if (round == 0) {
    CK(cudaMemsetAsync(c, 0, sizeof *c, st));
    CK(cudaMemsetAsync(b.bm, 0xff, sizeof(unsigned long long) * nq * b.plan_bm_cap, st));
    // 1. approximate leaves, grouping
    CK(hg::launch_route_queries(b.qin, (int)nq, (int)L, index_tree(ix), b.approx, st, b.bucket_cnt, nq,
                                prune ? b.leaf_cnt : nullptr, prune ? (uint32_t)nl : 0u, c->stamps + 0));
    CK(hg::launch_group_queries(b.approx, (int)nq, b.leaf_plan, nl, ix->tune.bound_tiles_per_item, b.qperm, b.slots,
                                b.leaf_qoff, b.leaf_qcnt, b.item_off, c->ctrl + 0, b.items, b.items_cap, st,
                                b.group_cnt));
    CK(hg::launch_rows_to_bf16(b.qin, b.qperm, nq, (int)L, b.qbf, b.qmeta, st));
    // 2. bound pass
    g.qperm = b.qperm;
    g.mode = 0;
    g.qtile = hg::kBatchQueryTile;
    g.items = b.items;
    g.nitems = b.items_cap;
    g.nitems_dev = c->ctrl + 0;
    g.queue = c->queues + 0;
    CK(hg::launch_umma_filter(ix->bd.rows_map, qmaps, g, sms, st));
    CK(hg::launch_bound_select(r, st));
    n_launch += 6;  // route, group (2), conversion, bound pass, bound selection
    // 3a. the leaves each query must filter (LB_EAPCA within B_q)
    if (prune) {
      CK(hg::launch_leaf_keep(b.qin, (int)L, (int)nq, b.useg_start, b.useg_end, b.nu, b.segstats, d.leaf_seg_off,
                              d.leaf_points, b.seg_uid, d.leaf_sk, d.leaf_size, nl, b.bound, b.leaf_cnt, b.leaf_q,
                              b.prune_nq, st));
      n_launch += 2;
    }
  } else {
    CK(cudaMemsetAsync(b.bucket_cnt, 0, sizeof(uint32_t) * nq, st));
    CK(cudaMemsetAsync(c->heads + 1, 0, sizeof(uint32_t), st));
    CK(hg::launch_rows_to_bf16(b.qin, list, nq, (int)L, b.qbf, b.qmeta, st, n_dev));
    ++n_launch;
    // a retry round prunes leaves again for its queries, against the bounds
    // the previous round lowered (a subset of the leaves kept before)
    if (prune) {
      CK(cudaMemsetAsync(b.leaf_cnt, 0, sizeof(uint32_t) * nl, st));
      CK(hg::launch_leaf_keep_list(b.segstats, b.nu, (int)L, (int)nq, d.leaf_seg_off, d.leaf_points, b.seg_uid,
                                   d.leaf_sk, d.leaf_size, nl, b.bound, b.leaf_cnt, b.leaf_q, b.prune_nq, list, n_dev,
                                   st));
      ++n_launch;
    }
  }
  // 3b. each leaf's queries laid out contiguously in a BF16 panel, and the
  // work items
  if (prune) {
    CK(hg::launch_group_pruned(b.leaf_cnt, b.leaf_q, b.prune_nq, b.leaf_plan, nl, ix->tune.filter_tiles_per_item,
                               tpi_min, b.panel_cap, b.items3_cap, nq, b.leaf_poff, b.leaf_ioff, pctl,
                               c->pairs + (round == 0 ? 0 : 1), b.panel_list, b.items3, st, n_dev));
    CK(hg::launch_rows_to_bf16(b.qin, b.panel_list, b.panel_cap, (int)L, b.panel_bf, nullptr, st, pctl + 1));
    n_launch += 3;
  }
  // 3c-5. certified filter, exact re-rank, verification; queries whose bucket
  // overflowed are retried with the bound their first survivors gave.  The
  // screening passes run on CTA pairs (cta_group::2) where the query tile
  // stays resident (L <= 256) unless the tuning asks for one CTA per tile.
  const bool pair = ix->tune.filter_cta_pair != 2 && L <= 256;  // four resident 64-column K blocks
  auto screen = [&](const hg::QueryMaps& q) {
    ++n_launch;
    return pair ? hg::launch_umma_pair(ix->bd.rows_map, q.q128, g, sms, st)
                : hg::launch_umma_filter(ix->bd.rows_map, q, g, sms, st);
  };
  g.errstat = round == 0 ? c->errstat : nullptr;
  g.stamp = c->stamps + 2 + 3 * round;
  if (prune) {
    g.mode = 3;
    g.items = b.items3;
    g.nitems = b.items3_cap;
    g.nitems_dev = pctl + 0;
    g.qperm = b.panel_list;
    g.nq_dev = nullptr;
    g.qtile = hg::kBatchQueryTile;
    g.queue = round == 0 ? c->queues + 1 : c->queues + 5 + round;
    CK(screen(b.panel_maps));
    g.stamp = nullptr;
  }
  // every row against every query: without pruning, and behind it where the
  // panel may overflow (its query count is then the round's, else 0)
  if (!prune || (uint64_t)b.panel_cap < (uint64_t)nl * nq) {
    g.mode = 1;
    g.qperm = round == 0 ? b.qperm : list;
    g.nq_dev = prune ? pctl + 2 : n_dev;
    g.qtile = round == 0 ? hg::kBatchQueryTile : 0;
    g.queue = c->queues + 2 + round;
    CK(screen(qmaps));
  }
  CK(hg::launch_scatter_pairs(b.pairs, c->heads + 1, b.pairs_cap, b.bucket, b.bucket_cnt, bucket_cap, nq,
                              c->stamps + 3 + 3 * round, st));
  CK(hg::launch_rerank(r, sms * (int)ix->tune.rerank_blocks_per_sm, st));
  CK(hg::launch_collect_retry(b.ok, list, nq, n_dev, lists[round & 1], c->ctrl + 4 + round + 1, c->ctrl + 3,
                              c->stamps + 4 + 3 * round, st));
  n_launch += 5;  // scatter, re-rank plan / segments / merge, collection
  *launches = n_launch;
  return HG_OK;
}

// A batch whose kmax is above kMaxK (the batched filter ranks at most
// kMaxK rows per query for its bound): every query through the plain path,
// in rounds above kMaxK, into the nq x kmax layout of the batched entry
// points (entries past a query's own k are +inf / -1).
static hg_status knn_batch_plain(hg_index* ix, const float* Q, uint32_t nq, const std::vector<uint32_t>& kq,
                                 uint32_t kmax, const hg_knn_opts& o, float* dist, int64_t* id, cudaStream_t st,
                                 hg_query_stats* stats, bool host_io) {
  CK(cudaSetDevice(ix->device));
  if (!st) st = ix->stream;
  const uint32_t L = ix->L;
  float* dq = const_cast<float*>(Q);
  float* dd = dist;
  int64_t* di = id;
  if (host_io) {
    CK(dalloc(&dq, (size_t)nq * L));
    cudaError_t e = dalloc(&dd, (size_t)nq * kmax);
    if (e == cudaSuccess) e = dalloc(&di, (size_t)nq * kmax);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dq, Q, sizeof(float) * nq * L, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) {
      dfree(dq);
      dfree(dd);
      dfree(di);
      return cuda_fail(e, "hg_knn_batch");
    }
  }
  hg_knn_opts po{};
  po.mode = HG_MODE_PLAIN;
  po.use_lb_sax = o.use_lb_sax;
  hg_status status = HG_OK;
  hg_query_stats acc{};
  for (uint32_t i = 0; i < nq && status == HG_OK; ++i) {
    hg_query_stats one{};
    status = knn_device_impl(ix, dq + (uint64_t)i * L, 1, kq[i], &po, dd + (uint64_t)i * kmax,
                             di + (uint64_t)i * kmax, st, &one);
    if (status == HG_OK && kq[i] < kmax) {
      cudaError_t e = cudaMemsetAsync(ix->s.topk_count, 0, sizeof(int), st);
      if (e == cudaSuccess)
        e = hg::launch_emit(ix->s.topk, ix->s.topk_count, (int)(kmax - kq[i]), dd + (uint64_t)i * kmax + kq[i],
                            di + (uint64_t)i * kmax + kq[i], st);
      if (e != cudaSuccess) status = cuda_fail(e, "hg_knn_batch");
    }
    acc.leaves_scanned += one.leaves_scanned;
    acc.rows_visited += one.rows_visited;
    acc.rows_lbsax_pruned += one.rows_lbsax_pruned;
    acc.chunks_loaded += one.chunks_loaded;
    acc.rows_completed += one.rows_completed;
    acc.rows_considered += one.rows_considered;
    acc.device_ms += one.device_ms;
    acc.fallback_ms += one.device_ms;
    acc.kernel_launches += one.kernel_launches + (kq[i] < kmax ? 1 : 0);
  }
  if (host_io) {
    if (status == HG_OK) {
      cudaError_t e = cudaMemcpyAsync(dist, dd, sizeof(float) * nq * kmax, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(id, di, sizeof(int64_t) * nq * kmax, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) status = cuda_fail(e, "hg_knn_batch");
    }
    dfree(dq);
    dfree(dd);
    dfree(di);
  }
  if (status == HG_OK && stats) {
    *stats = acc;
    stats->queries = nq;
    stats->fallback_queries = nq;
  }
  return status;
}

// Every buffer of a batch of nq queries with at most kmax answers each.
static hg_status ensure_batch_buffers(hg_index* ix, uint32_t nq, uint32_t kmax, uint32_t bucket_cap, bool want_prune,
                                      bool* prune, cudaStream_t st) {
  hg::BatchScratch& b = ix->bs;
  HCK(ensure_scratch(ix, 1, true));
  HCK(ensure_batch_data(ix, st));
  HCK(ensure_leaf_plan(ix, std::max<uint64_t>(2ull * kmax + 32, 256), st));
  const uint64_t items_cap =
      hg::bound_items_room(nq, ix->leaves.size(), b.plan_max_use, ix->tune.bound_tiles_per_item);
  if (items_cap > UINT32_MAX) return set_error(HG_ERR_NOMEM, "hg_knn_batch: bound pass work list");
  HCK(ensure_batch_scratch(ix, std::max(nq, b.nq_cap), bucket_cap, b.plan_bm_cap, (uint32_t)items_cap, kmax));
  if (!b.qlist2 || !b.qin || b.out_kmax < kmax) {
    dfree(b.qlist2);
    dfree(b.qin);
    dfree(b.out_dist);
    dfree(b.out_id);
    CK(dalloc(&b.qlist2, b.nq_cap));
    CK(dalloc(&b.qin, (size_t)b.nq_cap * ix->L));
    CK(dalloc(&b.out_dist, (size_t)b.nq_cap * kmax));
    CK(dalloc(&b.out_id, (size_t)b.nq_cap * kmax));
    b.out_kmax = kmax;
    ++b.gen;
  }
  if (want_prune) HCK(ensure_prune_scratch(ix, prune));
  return HG_OK;
}

// Batched exact k-NN; ks is a host array (or null).  Queries and answers are
// device buffers, or host buffers with host_io (copied straight into and out
// of the handle's fixed buffers: no allocation per call).
static hg_status knn_batch_impl(hg_index* ix, const float* d_Q, uint32_t nq, const uint32_t* ks, uint32_t kmax,
                                const hg_knn_opts& o, float* d_dist, int64_t* d_id, cudaStream_t st,
                                hg_query_stats* stats, bool host_io) {
  if (!ix || (!d_Q && nq)) return set_error(HG_ERR_ARG, "hg_knn_batch: null argument");
  if (kmax == 0) return set_error(HG_ERR_ARG, "hg_knn_batch: k must be positive");
  if (ix->L > 16384) return set_error(HG_ERR_LIMIT, "hg_knn_batch: series longer than 16384");
  if (nq > (1u << 24)) return set_error(HG_ERR_LIMIT, "hg_knn_batch: more than 2^24 queries");
  if ((int)kmax > hg::kMaxK) {
    std::vector<uint32_t> kq(nq, kmax);
    if (ks)
      for (uint32_t i = 0; i < nq; ++i) {
        if (ks[i] == 0 || ks[i] > kmax) return set_error(HG_ERR_ARG, "hg_knn_batch: ks[i] outside 1..kmax");
        kq[i] = ks[i];
      }
    if (stats) memset(stats, 0, sizeof *stats);
    if (nq == 0) return HG_OK;
    return knn_batch_plain(ix, d_Q, nq, kq, kmax, o, d_dist, d_id, st, stats, host_io);
  }
  if (!host_io && ((uintptr_t)d_Q & 15) != 0)
    return set_error(HG_ERR_ARG, "hg_knn_batch: queries must be 16-byte aligned");
  std::vector<uint32_t> kq(nq, kmax);
  if (ks)
    for (uint32_t i = 0; i < nq; ++i) {
      if (ks[i] == 0 || ks[i] > kmax) return set_error(HG_ERR_ARG, "hg_knn_batch: ks[i] outside 1..kmax");
      kq[i] = ks[i];
    }
  if (stats) memset(stats, 0, sizeof *stats);
  if (nq == 0) return HG_OK;
  CK(cudaSetDevice(ix->device));
  if (!st) st = ix->stream;
  const bool data_built = ix->bd.xbf == nullptr;
  const uint32_t L = ix->L;
  const uint32_t bucket_cap = o.bucket_cap > 0 ? (uint32_t)o.bucket_cap : kDefaultBucket;
  hg::BatchScratch& b = ix->bs;
  bool prune = false;
  hg_status bst = ensure_batch_buffers(ix, nq, kmax, bucket_cap, o.dense_filter == 0, &prune, st);
  hg::HostIo& io = ix->io;
  const bool own_io = d_Q != io.q && io.q_cap + io.out_cap > 0;
  if (bst == HG_ERR_NOMEM && (std::max(ix->s.slots, ix->s.list_slots) > 1 || own_io)) {
    // the scratch of an earlier plain call's groups (lists of 4 GB at most) and
    // its copies of queries and answers may hold what the batch lacks
    free_batch_scratch(b);
    free_scratch(ix);
    free_lists(ix);
    if (own_io) trim_io(io, 0);
    bst = ensure_batch_buffers(ix, nq, kmax, bucket_cap, o.dense_filter == 0, &prune, st);
  }
  if (bst != HG_OK) {
    // sets that are half there, or sized for a batch that did not fit, must not
    // meet the next call
    free_batch_scratch(b);
    return bst;
  }
  // inputs at fixed addresses: the queries and their k
  CK(cudaMemcpyAsync(b.qin, d_Q, sizeof(float) * nq * L,
                     host_io ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
  CK(cudaMemcpyAsync(b.kq, kq.data(), sizeof(uint32_t) * nq, cudaMemcpyHostToDevice, st));
  // the rounds, each captured once per shape in a CUDA graph and replayed
  const uint64_t key[8] = {nq, kmax, bucket_cap, b.gen, ix->tune.filter_tiles_per_item, ix->tune.bound_tiles_per_item,
                           ix->tune.rerank_blocks_per_sm, (prune ? 2u : 1u) | (ix->tune.filter_cta_pair << 4)};
  if (memcmp(key, b.graph_key, sizeof key) != 0) {
    drop_graphs(b);
    memcpy(b.graph_key, key, sizeof key);
  }
  uint64_t launches = 0;
  hg::BatchCtl hc;
  int round = 0;
  auto copy_answers = [&]() -> hg_status {
    const cudaMemcpyKind kind = host_io ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (d_dist) CK(cudaMemcpyAsync(d_dist, b.out_dist, sizeof(float) * nq * kmax, kind, st));
    if (d_id) CK(cudaMemcpyAsync(d_id, b.out_id, sizeof(int64_t) * nq * kmax, kind, st));
    return HG_OK;
  };
  for (;; ++round) {
    if (!b.graph[round]) {
      hg::QueryMaps qmaps;
      HCK(encode_query_maps(&qmaps, b.qbf, nq, L));
      cudaGraph_t graph = nullptr;
      CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed));
      const hg_status s = enqueue_round(ix, round, nq, kmax, bucket_cap, qmaps, prune, st, &b.graph_launches[round]);
      const cudaError_t ce = cudaStreamEndCapture(st, &graph);
      if (s != HG_OK) {
        if (graph) cudaGraphDestroy(graph);
        return s;
      }
      CK(ce);
      const cudaError_t ie = cudaGraphInstantiate(&b.graph[round], graph, 0);
      cudaGraphDestroy(graph);
      if (ie != cudaSuccess) b.graph[round] = nullptr;
      CK(ie);
    }
    launches += b.graph_launches[round];
    CK(cudaGraphLaunch(b.graph[round], st));
    // the answers with the counters, before the round's one synchronisation:
    // nearly always they are final
    HCK(copy_answers());
    CK(cudaMemcpyAsync(&hc, b.ctl, sizeof hc, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    // the queries left to retry, while rounds are left
    if (hc.heads[3] || round == kBatchRetries || hc.ctrl[4 + round + 1] == 0) break;
  }
  const uint32_t dev_err = hc.heads[3], *ctrl = hc.ctrl, *pc = hc.pctl;
  const unsigned long long *hs = hc.stats, *ts = hc.stamps;
  const double* es = hc.errstat;
  const uint32_t unverified = ctrl[3] + ctrl[4 + round + 1];
  if (dev_err) return set_error(HG_ERR_TIMEOUT, "hg_knn_batch: a tensor-core filter wait timed out");
  // queries that did not verify: the plain path
  uint64_t fallbacks = 0, fallback_launches = 0;
  float tf = 0;
  if (unverified > 0) {
    for (cudaEvent_t& e : ix->ev)
      if (!e) CK(cudaEventCreate(&e));
    std::vector<int> ok(nq);
    CK(cudaMemcpyAsync(ok.data(), b.ok, sizeof(int) * nq, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    hg_knn_opts po{};
    po.mode = HG_MODE_PLAIN;
    po.use_lb_sax = 1;
    // in groups of equal k, gathered from the batch: an approximate leaf of few
    // more rows than k leaves many queries without a bound (512 queries of 1M x
    // 256, leaf 1,500, k = 100: 145 of them, 18.8 ms one by one, 5.3 in groups)
    std::vector<uint32_t> left;
    for (uint32_t q = 0; q < nq; ++q)
      if (ok[q] != 1) left.push_back(q);
    std::stable_sort(left.begin(), left.end(), [&](uint32_t x, uint32_t y) { return kq[x] < kq[y]; });
    fallbacks = left.size();
    HCK(ensure_scratch(ix, group_slots(ix, (uint32_t)fallbacks), true));
    CK(cudaMemsetAsync(ix->s.err, 0, sizeof(int), st));
    CK(cudaEventRecord(ix->ev[0], st));
    for (size_t i = 0, n; i < left.size(); i += n) {
      const int k = (int)kq[left[i]];
      const size_t most = std::min<size_t>(left.size() - i, group_room(ix, true));
      for (n = 1; n < most && (int)kq[left[i + n]] == k;) ++n;
      const uint32_t q = left[i];
      if (n == 1) {
        HCK(knn_group(ix, b.qin + (uint64_t)q * L, 1, k, po, b.out_dist + (uint64_t)q * kmax,
                      b.out_id + (uint64_t)q * kmax, st, nullptr, &fallback_launches));
        continue;
      }
      CK(cudaMemcpyAsync(ix->s.group_row, left.data() + i, sizeof(uint32_t) * n, cudaMemcpyHostToDevice, st));
      CK(hg::launch_gather_rows(b.qin, (int)L, ix->s.group_row, n, ix->s.group_q, st));
      ++fallback_launches;
      HCK(knn_group(ix, ix->s.group_q, (int)n, k, po, b.out_dist, b.out_id, st, nullptr, &fallback_launches, false, 0.0f,
                    ix->s.group_row, kmax));
    }
    CK(cudaEventRecord(ix->ev[1], st));
    HCK(copy_answers());
    int ferr = 0;
    CK(cudaMemcpyAsync(&ferr, ix->s.err, sizeof ferr, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (ferr) return set_error(HG_ERR_TIMEOUT, "hg_knn_batch: an LB_SAX filter wait timed out");
    cudaEventElapsedTime(&tf, ix->ev[0], ix->ev[1]);
  }
  if (stats) {
    auto span = [&](int i, int j) { return (double)(ts[j] - ts[i]) * 1e-6; };  // ms
    double gemm = 0, rerank = 0;
    uint64_t pairs = 0, retried = 0;
    const double t01 = span(0, 2);
    for (int i = 0; i <= round; ++i) {
      const uint64_t cnt = i == 0 ? nq : ctrl[4 + i];
      if (i > 0) retried += cnt;
      gemm += span(2 + 3 * i, 3 + 3 * i);
      rerank += span(3 + 3 * i, 4 + 3 * i);
      // the first filter round with pruning: the kept pairs, plus every pair if the dense
      // pass ran instead
      pairs += (i == 0 && prune) ? hc.pairs[0] + (uint64_t)pc[2] * ix->n : cnt * ix->n;
    }
    const double t0e = span(0, 4 + 3 * round) + (fallbacks ? tf : 0.0);
    stats->queries = nq;
    stats->rows_visited = hs[0];
    stats->chunks_loaded = hs[1];
    stats->survivors = hs[2];
    stats->bf16_pairs = pairs;
    stats->fallback_queries = fallbacks;
    stats->retried_queries = retried;
    stats->bound_ms = t01;
    stats->gemm_ms = gemm;
    stats->rerank_ms = rerank;
    stats->fallback_ms = fallbacks ? tf : 0.0;
    stats->device_ms = t0e;
    stats->kernel_launches = launches + (data_built ? 2 : 0) + fallback_launches;
    stats->err_mean = es[2] > 0 ? es[0] / es[2] : 0.0;
    stats->err_max = es[4];
    stats->err_over_bound = es[3] > 0 ? es[1] / es[3] : 0.0;
    uint64_t nonempty = 0;
    for (int l : ix->leaves) nonempty += ix->nodes[l].node_size > 0 ? 1 : 0;
    stats->leaf_pairs = prune ? (uint64_t)nq * nonempty : 0;
    stats->leaf_pairs_kept = prune ? pc[3] : 0;
  }
  return HG_OK;
}

// ---------------------------------------------------------------------------
// host generators (same bits as the kernels)
// ---------------------------------------------------------------------------

template <class F>
static void parallel_for(uint64_t n, F f) {
  unsigned nt = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
  if (n < 64) nt = 1;
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nt; ++t)
    th.emplace_back([=]() {
      for (uint64_t i = t; i < n; i += nt) f(i);
    });
  for (auto& x : th) x.join();
}

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

extern "C" {

const char* hg_status_string(hg_status s) {
  switch (s) {
    case HG_OK: return "ok";
    case HG_ERR_ARG: return "invalid argument";
    case HG_ERR_IO: return "i/o error";
    case HG_ERR_FORMAT: return "index format error";
    case HG_ERR_CUDA: return "CUDA error";
    case HG_ERR_NOMEM: return "out of memory";
    case HG_ERR_TIMEOUT: return "device wait timed out";
    case HG_ERR_LIMIT: return "size limit exceeded";
    default: return "unknown status";
  }
}

const char* hg_last_error(void) { return g_last_error; }

hg_status hg_index_build(const float* data, int data_on_device, uint64_t n, uint32_t L, uint32_t leaf_size,
                         int device, hg_index** out) {
  return build_impl(data, data_on_device, n, L, leaf_size, device, out);
}

hg_status hg_index_build_file(const char* dataset, uint64_t n, uint32_t L, uint32_t leaf_size, int device,
                              hg_index** out) {
  if (!dataset || !out || L == 0) return set_error(HG_ERR_ARG, "hg_index_build_file: null argument");
  FILE* f = fopen(dataset, "rb");
  if (!f) return set_error(HG_ERR_IO, "hg_index_build_file: dataset not found");
  fseek(f, 0, SEEK_END);
  const uint64_t sz = (uint64_t)ftell(f);
  fseek(f, 0, SEEK_SET);
  if (sz / (sizeof(float) * L) < n) {
    fclose(f);
    return set_error(HG_ERR_IO, "hg_index_build_file: the file holds fewer series than requested");
  }
  std::vector<float> buf;
  try {
    buf.resize((size_t)n * L);
  } catch (...) {
    fclose(f);
    return set_error(HG_ERR_NOMEM, "hg_index_build_file: host allocation");
  }
  const size_t got = fread(buf.data(), sizeof(float) * L, n, f);
  fclose(f);
  if (got != n) return set_error(HG_ERR_IO, "hg_index_build_file: short read");
  return build_impl(buf.data(), 0, n, L, leaf_size, device, out);
}

hg_status hg_index_write(hg_index* ix, const char* dir, double buffer_mb) { return write_impl(ix, dir, buffer_mb); }

hg_status hg_index_read(const char* dir, int device, hg_index** out) { return read_impl(dir, device, out); }

void hg_index_destroy(hg_index* ix) {
  if (!ix) return;
  cudaSetDevice(ix->device);
  free_device(ix);
  if (ix->stream) cudaStreamDestroy(ix->stream);
  delete ix;
}

hg_status hg_index_info_get(const hg_index* ix, hg_index_info* info) {
  if (!ix || !info) return set_error(HG_ERR_ARG, "hg_index_info_get: null argument");
  info->num_series = ix->n;
  info->ts_length = ix->L;
  info->leaf_size = ix->leaf_size;
  info->num_leaves = (uint32_t)ix->leaves.size();
  info->num_nodes = (uint32_t)ix->nodes.size();
  info->max_segments = (uint32_t)ix->max_seg;
  info->has_ids = ix->has_ids ? 1 : 0;
  info->device_bytes = (uint64_t)ix->n * ix->L * 4 + ix->n * (8 + 16);
  return HG_OK;
}

hg_status hg_index_leaf(const hg_index* ix, uint32_t i, uint64_t* file_pos, uint32_t* size, uint32_t* nseg) {
  if (!ix || i >= ix->leaves.size()) return set_error(HG_ERR_ARG, "hg_index_leaf: bad leaf");
  const Node& n = ix->nodes[ix->leaves[i]];
  if (file_pos) *file_pos = n.file_pos;
  if (size) *size = n.node_size;
  if (nseg) *nseg = (uint32_t)n.points.size();
  return HG_OK;
}

hg_status hg_index_leaf_envelope(const hg_index* ix, uint32_t i, short* points, float* env) {
  if (!ix || i >= ix->leaves.size()) return set_error(HG_ERR_ARG, "hg_index_leaf_envelope: bad leaf");
  const Node& n = ix->nodes[ix->leaves[i]];
  if (points) memcpy(points, n.points.data(), sizeof(short) * n.points.size());
  if (env) memcpy(env, n.sk.data(), sizeof(float) * n.sk.size());
  return HG_OK;
}

hg_status hg_index_row_ids(const hg_index* ix, int64_t* ids) {
  if (!ix || !ids) return set_error(HG_ERR_ARG, "hg_index_row_ids: null argument");
  memcpy(ids, ix->ids.data(), sizeof(int64_t) * ix->n);
  return HG_OK;
}

hg_status hg_index_rows(const hg_index* ix, uint64_t first, uint64_t count, float* rows, uint8_t* sax) {
  if (!ix || first + count > ix->n) return set_error(HG_ERR_ARG, "hg_index_rows: range outside the index");
  if (count == 0) return HG_OK;
  CK(cudaSetDevice(ix->device));
  if (rows) CK(cudaMemcpy(rows, ix->d.rows + first * ix->L, sizeof(float) * count * ix->L, cudaMemcpyDeviceToHost));
  if (sax) CK(cudaMemcpy(sax, ix->d.sax + first * 16, count * 16, cudaMemcpyDeviceToHost));
  return HG_OK;
}

hg_status hg_knn_device(hg_index* ix, const float* d_queries, uint32_t nq, uint32_t k, const hg_knn_opts* opts,
                        float* d_dist_out, int64_t* d_id_out, void* stream, hg_query_stats* stats) {
  return knn_device_impl(ix, d_queries, nq, k, opts, d_dist_out, d_id_out, (cudaStream_t)stream, stats);
}

hg_status hg_knn(hg_index* ix, const float* queries, uint32_t nq, uint32_t k, const hg_knn_opts* opts,
                 float* dist_out, int64_t* id_out, uint64_t* leaf_pos_out, hg_query_stats* stats) {
  if (!ix || (!queries && nq)) return set_error(HG_ERR_ARG, "hg_knn: null argument");
  if (nq == 0) return HG_OK;
  CK(cudaSetDevice(ix->device));
  const size_t nk = (size_t)nq * k, q_bytes = sizeof(float) * nq * ix->L, id_bytes = sizeof(int64_t) * nk;
  const size_t out_bytes = id_bytes + sizeof(float) * nk;
  hg::HostIo& io = ix->io;
  hg_status s = grow_io(&io.q, &io.q_cap, q_bytes);
  if (s == HG_OK) s = grow_io(&io.out, &io.out_cap, out_bytes);
  if (s != HG_OK) {
    trim_io(io, 0);
    return s;
  }
  // ids and distances side by side: one copy back
  int64_t* d_id = reinterpret_cast<int64_t*>(io.out);
  float* d_dist = reinterpret_cast<float*>(io.out + id_bytes);
  std::vector<int64_t> ids(nk + (nk + 1) / 2);
  const cudaError_t e = cudaMemcpyAsync(io.q, queries, q_bytes, cudaMemcpyHostToDevice, ix->stream);
  if (e != cudaSuccess) s = cuda_fail(e, "hg_knn");
  const bool batch = opts && opts->mode == HG_MODE_BATCH;
  if (s == HG_OK)
    s = knn_device_impl(ix, io.q, nq, k, opts, d_dist, d_id, ix->stream, stats, batch ? nullptr : ids.data(), io.out,
                        out_bytes);
  if (s == HG_OK && batch) {
    cudaError_t ce = cudaMemcpyAsync(ids.data(), io.out, out_bytes, cudaMemcpyDeviceToHost, ix->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(ix->stream);
    if (ce != cudaSuccess) s = cuda_fail(ce, "hg_knn");
  }
  trim_io(io, kHostIoKeep);
  if (s != HG_OK) return s;
  if (dist_out) memcpy(dist_out, ids.data() + nk, sizeof(float) * nk);
  if (id_out) memcpy(id_out, ids.data(), sizeof(int64_t) * nq * k);
  if (leaf_pos_out) {
    // answer id -> leaf-ordered row -> its leaf's file_pos
    std::vector<uint64_t> row_of_id;
    if (ix->has_ids) {
      row_of_id.assign(ix->n, 0);
      for (uint64_t r = 0; r < ix->n; ++r)
        if ((uint64_t)ix->ids[r] < ix->n) row_of_id[ix->ids[r]] = r;
    }
    std::vector<uint64_t> starts(ix->leaves.size());
    for (size_t i = 0; i < ix->leaves.size(); ++i) starts[i] = ix->nodes[ix->leaves[i]].file_pos;
    for (size_t j = 0; j < (size_t)nq * k; ++j) {
      if (ids[j] < 0) {
        leaf_pos_out[j] = UINT64_MAX;
        continue;
      }
      const uint64_t row = ix->has_ids ? row_of_id[ids[j]] : (uint64_t)ids[j];
      size_t li = std::upper_bound(starts.begin(), starts.end(), row) - starts.begin();
      // skip empty leaves sharing the start position
      while (li > 0 && ix->nodes[ix->leaves[li - 1]].node_size == 0) --li;
      leaf_pos_out[j] = li > 0 ? starts[li - 1] : 0;
    }
  }
  return HG_OK;
}

hg_status hg_knn_batch_device(hg_index* ix, const float* d_queries, uint32_t nq, const uint32_t* ks, uint32_t kmax,
                              const hg_knn_opts* opts, float* d_dist_out, int64_t* d_id_out, void* stream,
                              hg_query_stats* stats) {
  if (!d_dist_out || !d_id_out) return set_error(HG_ERR_ARG, "hg_knn_batch_device: null output");
  hg_knn_opts o{};
  if (opts) o = *opts;
  return knn_batch_impl(ix, d_queries, nq, ks, kmax, o, d_dist_out, d_id_out, (cudaStream_t)stream, stats);
}

hg_status hg_knn_batch(hg_index* ix, const float* queries, uint32_t nq, const uint32_t* ks, uint32_t kmax,
                       const hg_knn_opts* opts, float* dist_out, int64_t* id_out, hg_query_stats* stats) {
  if (!ix || (!queries && nq)) return set_error(HG_ERR_ARG, "hg_knn_batch: null argument");
  hg_knn_opts o{};
  if (opts) o = *opts;
  return knn_batch_impl(ix, queries, nq, ks, kmax, o, dist_out, id_out, nullptr, stats, true);
}

static hg_status bf16_dots_impl(const float* d_rows, uint64_t n, uint32_t L, const float* d_queries, uint32_t nq,
                                float* d_dots, void* stream, uint64_t wait_ns, int withhold) {
  if (!d_rows || !d_queries || !d_dots) return set_error(HG_ERR_ARG, "hg_bf16_dots: null argument");
  if (n == 0 || nq == 0) return HG_OK;
  if (L == 0 || L % 16 != 0 || L > 16384) return set_error(HG_ERR_ARG, "hg_bf16_dots: L must be a multiple of 16");
  if (n >= (1ull << 31) || nq >= (1u << 24)) return set_error(HG_ERR_LIMIT, "hg_bf16_dots: too many rows");
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  uint16_t* xbf = nullptr;
  uint16_t* qbf = nullptr;
  float4* xmeta = nullptr;
  float4* qmeta = nullptr;
  float4* tmeta = nullptr;
  uint32_t* perm = nullptr;
  int* err = nullptr;
  auto release = [&]() {
    dfree(xbf);
    dfree(qbf);
    dfree(xmeta);
    dfree(qmeta);
    dfree(tmeta);
    dfree(perm);
    dfree(err);
  };
  std::vector<uint32_t> ident(nq);
  for (uint32_t i = 0; i < nq; ++i) ident[i] = i;
  cudaError_t e = dalloc(&xbf, n * L);
  if (e == cudaSuccess) e = dalloc(&qbf, (size_t)nq * L);
  if (e == cudaSuccess) e = dalloc(&xmeta, n);
  if (e == cudaSuccess) e = dalloc(&qmeta, nq);
  if (e == cudaSuccess) e = dalloc(&tmeta, (n + 127) / 128);
  if (e == cudaSuccess) e = dalloc(&perm, nq);
  if (e == cudaSuccess) e = dalloc(&err, 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(perm, ident.data(), sizeof(uint32_t) * nq, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e == cudaSuccess) e = hg::launch_rows_to_bf16(d_rows, nullptr, n, (int)L, xbf, xmeta, st);
  if (e == cudaSuccess) e = hg::launch_rows_to_bf16(d_queries, nullptr, nq, (int)L, qbf, qmeta, st);
  if (e == cudaSuccess) e = hg::launch_tile_norms(xmeta, n, tmeta, st);
  if (e != cudaSuccess) {
    release();
    return cuda_fail(e, "hg_bf16_dots");
  }
  CUtensorMap xmap;
  hg::QueryMaps qmaps;
  hg_status hs = encode_bf16_map(&xmap, xbf, n, L, 128);
  if (hs == HG_OK) hs = encode_query_maps(&qmaps, qbf, nq, L);
  if (hs != HG_OK) {
    release();
    return hs;
  }
  hg::BatchGemm g{};
  g.L = (int)L;
  g.nrows = n;
  g.xmeta = xmeta;
  g.tile_meta = tmeta;
  g.qmeta = qmeta;
  g.qperm = perm;
  g.nq = (int)nq;
  g.mode = 2;
  g.qtile = nq <= 64 ? 64 : (nq <= 128 ? 128 : hg::kBatchQueryTile);
  g.tiles_per_item = 8;
  g.err = err;
  g.dots = d_dots;
  g.dots_ld = n;
  g.wait_ns = wait_ns;
  g.withhold_first_copy = withhold;
  e = hg::launch_umma_filter(xmap, qmaps, g, hg::sm_count(dev), st);
  int herr = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof herr, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  release();
  if (e != cudaSuccess) return cuda_fail(e, "hg_bf16_dots");
  if (herr) return set_error(HG_ERR_TIMEOUT, "hg_bf16_dots: a tensor-core wait timed out");
  return HG_OK;
}

hg_status hg_bf16_dots(const float* d_rows, uint64_t n, uint32_t L, const float* d_queries, uint32_t nq,
                       float* d_dots, void* stream) {
  return bf16_dots_impl(d_rows, n, L, d_queries, nq, d_dots, stream, 0, 0);
}

hg_status hg_filter_wait_check(uint32_t wait_us, int withhold, void* stream) {
  if (wait_us == 0 || wait_us > 2000000u) return set_error(HG_ERR_ARG, "hg_filter_wait_check: wait_us outside 1..2e6");
  cudaStream_t st = (cudaStream_t)stream;
  constexpr uint64_t n = 512;
  constexpr uint32_t L = 64, nq = 64;
  float* rows = nullptr;
  float* qs = nullptr;
  float* dots = nullptr;
  cudaError_t e = dalloc(&rows, n * L);
  if (e == cudaSuccess) e = dalloc(&qs, (size_t)nq * L);
  if (e == cudaSuccess) e = dalloc(&dots, n * nq);
  if (e == cudaSuccess) e = hg::launch_generate_walks(1, 0, n, (int)L, rows, st, 0);
  if (e == cudaSuccess) e = hg::launch_generate_walks(2, 0, nq, (int)L, qs, st, 0);
  hg_status hs = e == cudaSuccess ? HG_OK : cuda_fail(e, "hg_filter_wait_check");
  if (hs == HG_OK) hs = bf16_dots_impl(rows, n, L, qs, nq, dots, stream, (uint64_t)wait_us * 1000ull, withhold ? 1 : 0);
  dfree(rows);
  dfree(qs);
  dfree(dots);
  return hs;
}

// The CTA-pair filter (k_umma_pair, mode 1) once over n rows x nq queries
// with every bound +inf (no survivors), each bounded wait shortened to
// wait_ns; withhold = 1 leaves out the odd CTA's first row copy, so the
// leader's barrier phase never completes.
static hg_status pair_wait_impl(const float* d_rows, uint64_t n, uint32_t L, const float* d_queries, uint32_t nq,
                                cudaStream_t st, uint64_t wait_ns, int withhold) {
  uint16_t* xbf = nullptr;
  uint16_t* qbf = nullptr;
  float4* xmeta = nullptr;
  float4* qmeta = nullptr;
  float4* tmeta = nullptr;
  uint32_t* perm = nullptr;
  float* bound = nullptr;
  unsigned long long* pairs = nullptr;
  uint32_t* cnt = nullptr;
  int* err = nullptr;
  auto release = [&]() {
    dfree(xbf);
    dfree(qbf);
    dfree(xmeta);
    dfree(qmeta);
    dfree(tmeta);
    dfree(perm);
    dfree(bound);
    dfree(pairs);
    dfree(cnt);
    dfree(err);
  };
  constexpr uint32_t kPairsCap = 4096;
  std::vector<uint32_t> ident(nq);
  std::vector<float> inf(nq, INFINITY);
  for (uint32_t i = 0; i < nq; ++i) ident[i] = i;
  cudaError_t e = dalloc(&xbf, n * L);
  if (e == cudaSuccess) e = dalloc(&qbf, (size_t)nq * L);
  if (e == cudaSuccess) e = dalloc(&xmeta, n);
  if (e == cudaSuccess) e = dalloc(&qmeta, nq);
  if (e == cudaSuccess) e = dalloc(&tmeta, (n + 127) / 128);
  if (e == cudaSuccess) e = dalloc(&perm, nq);
  if (e == cudaSuccess) e = dalloc(&bound, nq);
  if (e == cudaSuccess) e = dalloc(&pairs, kPairsCap);
  if (e == cudaSuccess) e = dalloc(&cnt, 1);
  if (e == cudaSuccess) e = dalloc(&err, 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(perm, ident.data(), sizeof(uint32_t) * nq, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(bound, inf.data(), sizeof(float) * nq, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(uint32_t), st);
  if (e == cudaSuccess) e = hg::launch_rows_to_bf16(d_rows, nullptr, n, (int)L, xbf, xmeta, st);
  if (e == cudaSuccess) e = hg::launch_rows_to_bf16(d_queries, nullptr, nq, (int)L, qbf, qmeta, st);
  if (e == cudaSuccess) e = hg::launch_tile_norms(xmeta, n, tmeta, st);
  if (e != cudaSuccess) {
    release();
    return cuda_fail(e, "hg_filter_pair_wait_check");
  }
  CUtensorMap xmap, qmap;
  hg_status hs = encode_bf16_map(&xmap, xbf, n, L, 128);
  if (hs == HG_OK) hs = encode_bf16_map(&qmap, qbf, nq, L, hg::kBatchQueryTile / 2);
  if (hs != HG_OK) {
    release();
    return hs;
  }
  hg::BatchGemm g{};
  g.L = (int)L;
  g.nrows = n;
  g.xmeta = xmeta;
  g.tile_meta = tmeta;
  g.qmeta = qmeta;
  g.qperm = perm;
  g.nq = (int)nq;
  g.mode = 1;
  g.qtile = hg::kBatchQueryTile;
  g.tiles_per_item = 8;
  filter_coefficients(L, &g.c_acc, &g.c_sq);
  g.bound = bound;
  g.pairs = pairs;
  g.pairs_cnt = cnt;
  g.pairs_cap = kPairsCap;
  g.err = err;
  g.wait_ns = wait_ns;
  g.withhold_first_copy = withhold;
  int dev = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = hg::launch_umma_pair(xmap, qmap, g, hg::sm_count(dev), st);
  int herr = 0;
  uint32_t hcnt = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof herr, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hcnt, cnt, sizeof hcnt, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  release();
  if (e != cudaSuccess) return cuda_fail(e, "hg_filter_pair_wait_check");
  if (herr) return set_error(HG_ERR_TIMEOUT, "hg_filter_pair_wait_check: a tensor-core wait timed out");
  if (hcnt != 0) return set_error(HG_ERR_CUDA, "hg_filter_pair_wait_check: survivors without a bound");
  return HG_OK;
}

hg_status hg_filter_pair_wait_check(uint32_t wait_us, int withhold, void* stream) {
  if (wait_us == 0 || wait_us > 2000000u)
    return set_error(HG_ERR_ARG, "hg_filter_pair_wait_check: wait_us outside 1..2e6");
  cudaStream_t st = (cudaStream_t)stream;
  constexpr uint64_t n = 1024;
  constexpr uint32_t L = 64, nq = 64;
  float* rows = nullptr;
  float* qs = nullptr;
  cudaError_t e = dalloc(&rows, n * L);
  if (e == cudaSuccess) e = dalloc(&qs, (size_t)nq * L);
  if (e == cudaSuccess) e = hg::launch_generate_walks(1, 0, n, (int)L, rows, st, 0);
  if (e == cudaSuccess) e = hg::launch_generate_walks(2, 0, nq, (int)L, qs, st, 0);
  hg_status hs = e == cudaSuccess ? HG_OK : cuda_fail(e, "hg_filter_pair_wait_check");
  if (hs == HG_OK) hs = pair_wait_impl(rows, n, L, qs, nq, st, (uint64_t)wait_us * 1000ull, withhold ? 1 : 0);
  dfree(rows);
  dfree(qs);
  return hs;
}

hg_status hg_tuning_get(const hg_index* ix, hg_tuning* out) {
  if (!ix || !out) return set_error(HG_ERR_ARG, "hg_tuning_get: null argument");
  *out = ix->tune;
  return HG_OK;
}

hg_status hg_tuning_set(hg_index* ix, const hg_tuning* t) {
  if (!ix || !t) return set_error(HG_ERR_ARG, "hg_tuning_set: null argument");
  auto bad = [](uint32_t v, uint32_t lo, uint32_t hi) { return v != 0 && (v < lo || v > hi); };
  if (bad(t->filter_tiles_per_item, 8, 128) || bad(t->bound_tiles_per_item, 2, 64) ||
      bad(t->rerank_blocks_per_sm, 1, 16) || bad(t->approx_blocks_per_sm, 1, 4) || bad(t->filter_cta_pair, 1, 2))
    return set_error(HG_ERR_ARG, "hg_tuning_set: a parameter outside its range");
  if (t->filter_tiles_per_item) ix->tune.filter_tiles_per_item = t->filter_tiles_per_item;
  if (t->bound_tiles_per_item) ix->tune.bound_tiles_per_item = t->bound_tiles_per_item;
  if (t->rerank_blocks_per_sm) ix->tune.rerank_blocks_per_sm = t->rerank_blocks_per_sm;
  if (t->approx_blocks_per_sm) ix->tune.approx_blocks_per_sm = t->approx_blocks_per_sm;
  if (t->filter_cta_pair) ix->tune.filter_cta_pair = t->filter_cta_pair;
  return HG_OK;
}

// Coordinate descent over the launch parameters: each parameter in turn takes
// every candidate value with the others fixed, timed on the caller's queries
// (the batched call's device time from its %globaltimer stamps; the plain path
// on up to 64 of the queries, k <= 10); the fastest of two runs per value stays.
hg_status hg_autotune(hg_index* ix, const float* d_queries, uint32_t nq, const uint32_t* ks, uint32_t kmax,
                      void* stream, hg_tuning* out) {
  if (!ix || !d_queries || nq == 0 || kmax == 0) return set_error(HG_ERR_ARG, "hg_autotune: bad argument");
  CK(cudaSetDevice(ix->device));
  cudaStream_t st = stream ? (cudaStream_t)stream : ix->stream;
  float* d_dist = nullptr;
  int64_t* d_id = nullptr;
  CK(dalloc(&d_dist, (size_t)nq * kmax));
  cudaError_t e = dalloc(&d_id, (size_t)nq * kmax);
  if (e != cudaSuccess) {
    dfree(d_dist);
    return cuda_fail(e, "hg_autotune");
  }
  hg_knn_opts o{};
  hg_status status = HG_OK;
  auto batch_ms = [&](double* ms) -> hg_status {
    hg_query_stats sq;
    hg_status r = knn_batch_impl(ix, d_queries, nq, ks, kmax, o, d_dist, d_id, st, &sq);
    *ms = sq.device_ms;
    return r;
  };
  const uint32_t np = std::min<uint32_t>(nq, 64), kp = std::min<uint32_t>(kmax, 10);
  auto plain_ms = [&](double* ms) -> hg_status {
    hg_query_stats sq;
    hg_knn_opts po{};
    po.use_lb_sax = 1;
    hg_status r = knn_device_impl(ix, d_queries, np, kp, &po, d_dist, d_id, st, &sq);
    *ms = sq.device_ms;
    return r;
  };
  struct Param {
    uint32_t* field;
    std::vector<uint32_t> cand;
    bool plain;
  };
  hg_tuning& t = ix->tune;
  // (filter_cta_pair is not among them: the CTA-pair kernel was slower in
  // every measurement; it stays selectable through hg_tuning_set)
  std::vector<Param> params = {{&t.filter_tiles_per_item, {16, 32, 64}, false},
                               {&t.bound_tiles_per_item, {4, 8, 16}, false},
                               {&t.rerank_blocks_per_sm, {4, 8, 16}, false},
                               {&t.approx_blocks_per_sm, {1, 2, 4}, true}};
  double warm = 0;
  status = batch_ms(&warm);  // also builds the BF16 copy on a first call
  for (auto& p : params) {
    if (status != HG_OK) break;
    uint32_t best = *p.field;
    double best_ms = 1e30;
    for (uint32_t v : p.cand) {
      *p.field = v;
      double ms = 0, ms2 = 0;
      status = p.plain ? plain_ms(&ms) : batch_ms(&ms);
      if (status == HG_OK) status = p.plain ? plain_ms(&ms2) : batch_ms(&ms2);
      if (status != HG_OK) break;
      ms = std::min(ms, ms2);
      if (ms < best_ms) {
        best_ms = ms;
        best = v;
      }
    }
    *p.field = best;
    if (p.plain) t.plain_ms = best_ms;
    else t.batch_ms = best_ms;
  }
  dfree(d_dist);
  dfree(d_id);
  if (status != HG_OK) return status;
  if (out) *out = t;
  return HG_OK;
}

hg_status hg_route(hg_index* ix, const float* queries, uint32_t nq, int32_t* leaf_out) {
  if (!ix || !queries || !leaf_out) return set_error(HG_ERR_ARG, "hg_route: null argument");
  if (nq == 0) return HG_OK;
  CK(cudaSetDevice(ix->device));
  float* d_q = nullptr;
  int* d_l = nullptr;
  CK(dalloc(&d_q, (size_t)nq * ix->L));
  cudaError_t e = dalloc(&d_l, nq);
  if (e == cudaSuccess) e = cudaMemcpy(d_q, queries, sizeof(float) * nq * ix->L, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = hg::launch_route_queries(d_q, (int)nq, (int)ix->L, index_tree(ix), d_l, ix->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(leaf_out, d_l, sizeof(int) * nq, cudaMemcpyDeviceToHost, ix->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
  cudaFree(d_q);
  if (d_l) cudaFree(d_l);
  return e == cudaSuccess ? HG_OK : cuda_fail(e, "hg_route");
}

hg_status hg_leaf_lower_bounds(hg_index* ix, const float* query, float* lb_out) {
  if (!ix || !query || !lb_out) return set_error(HG_ERR_ARG, "hg_leaf_lower_bounds: null argument");
  CK(cudaSetDevice(ix->device));
  const int nl = (int)ix->leaves.size();
  float* d_q = nullptr;
  float* d_lb = nullptr;
  CK(dalloc(&d_q, ix->L));
  cudaError_t e = dalloc(&d_lb, nl);
  if (e == cudaSuccess) e = cudaMemcpy(d_q, query, sizeof(float) * ix->L, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    hg::PrepArgs p = prep_args(ix, d_q);
    p.approx_leaf = nullptr;  // lower bounds only
    p.lb = d_lb;
    e = hg::launch_query_prep(p, 1, ix->stream);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(lb_out, d_lb, sizeof(float) * nl, cudaMemcpyDeviceToHost, ix->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
  cudaFree(d_q);
  if (d_lb) cudaFree(d_lb);
  return e == cudaSuccess ? HG_OK : cuda_fail(e, "hg_leaf_lower_bounds");
}

static hg_status generate_rows(uint64_t seed, uint64_t first, uint64_t n, uint32_t L, float* out, int on_device,
                               int device, int unit) {
  if (!out || L == 0 || L % 4 != 0) return set_error(HG_ERR_ARG, "hg_generate_walks: L must be a multiple of 4");
  if (on_device) {
    CK(cudaSetDevice(device));
    CK(hg::launch_generate_walks(seed, first, n, (int)L, out, 0, unit));
    CK(cudaStreamSynchronize(0));
    return HG_OK;
  }
  parallel_for(n, [=](uint64_t i) {
    if (unit) hg::gaussian_unit(seed, first + i, (int)L, out + i * L);
    else hg::random_walk(seed, first + i, (int)L, out + i * L);
  });
  return HG_OK;
}

// data == nullptr: each base row is regenerated from data_seed (the rows
// of hg_generate_walks / hg_generate_unit_vectors with that seed).
static hg_status generate_queries(uint64_t seed, const float* data, uint64_t n, uint32_t L, uint32_t nq,
                                  const double* sigma2, float* out, uint64_t* base_ids, int on_device, int device,
                                  int unit, uint64_t data_seed = 0) {
  if (!out || !sigma2 || n == 0 || L == 0 || L % 4 != 0)
    return set_error(HG_ERR_ARG, "hg_generate_queries: bad argument");
  if (on_device) {
    CK(cudaSetDevice(device));
    double* d_s = nullptr;
    CK(dalloc(&d_s, nq));
    cudaError_t e = cudaMemcpy(d_s, sigma2, sizeof(double) * nq, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
      e = hg::launch_generate_queries(seed, data, n, (int)L, (int)nq, d_s, out, base_ids, 0, unit, data_seed);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    cudaFree(d_s);
    return e == cudaSuccess ? HG_OK : cuda_fail(e, "hg_generate_queries");
  }
  parallel_for(nq, [=](uint64_t j) {
    const uint64_t b = hg::pick_row(seed, j, n);
    if (base_ids) base_ids[j] = b;
    float* o = out + j * L;
    const float* base = data ? data + b * L : o;
    if (!data) {
      if (unit) hg::gaussian_unit(data_seed, b, (int)L, o);
      else hg::random_walk(data_seed, b, (int)L, o);
    }
    hg::noisy_query(seed, j, base, (int)L, sigma2[j], o, unit);
  });
  return HG_OK;
}

hg_status hg_generate_queries_seeded(uint64_t data_seed, uint64_t seed, uint64_t n, uint32_t L, uint32_t nq,
                                     const double* sigma2, int unit, float* out, uint64_t* base_ids, int on_device,
                                     int device) {
  return generate_queries(seed, nullptr, n, L, nq, sigma2, out, base_ids, on_device, device, unit ? 1 : 0,
                          data_seed);
}

hg_status hg_generate_walks(uint64_t seed, uint64_t first, uint64_t n, uint32_t L, float* out, int on_device,
                            int device) {
  return generate_rows(seed, first, n, L, out, on_device, device, 0);
}

hg_status hg_generate_queries(uint64_t seed, const float* data, uint64_t n, uint32_t L, uint32_t nq,
                              const double* sigma2, float* out, uint64_t* base_ids, int on_device, int device) {
  return generate_queries(seed, data, n, L, nq, sigma2, out, base_ids, on_device, device, 0);
}

hg_status hg_generate_unit_vectors(uint64_t seed, uint64_t first, uint64_t n, uint32_t L, float* out, int on_device,
                                   int device) {
  return generate_rows(seed, first, n, L, out, on_device, device, 1);
}

hg_status hg_generate_unit_queries(uint64_t seed, const float* data, uint64_t n, uint32_t L, uint32_t nq,
                                   const double* sigma2, float* out, uint64_t* base_ids, int on_device, int device) {
  return generate_queries(seed, data, n, L, nq, sigma2, out, base_ids, on_device, device, 1);
}

hg_status hg_sax_breakpoints(float* out255) {
  if (!out255) return set_error(HG_ERR_ARG, "hg_sax_breakpoints: null argument");
  memcpy(out255, kHgBreakpoints, sizeof(float) * 255);
  return HG_OK;
}

}  // extern "C"
