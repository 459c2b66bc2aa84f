// The network object: cfg parsing, weights loading and the forward loop for the
// layer types on the convolutional forward path.  Mirrors the reference's
// parse_network_cfg (src/parser.c:742-889), load_weights (src/parser.c:1218-1308),
// forward_network_gpu (src/network.c:762-788) and network_predict
// (src/network.c:497-508), with activations kept channels-last between layers.
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "common.h"
#include "conv.h"
#include "host_copy.h"

using namespace dnb;

namespace {

enum LayerKind { L_CONV, L_MAXPOOL, L_UPSAMPLE, L_SHORTCUT, L_ROUTE, L_YOLO, L_AVGPOOL, L_SOFTMAX, L_CONNECTED };
const char *const kKindNames[] = {"convolutional", "maxpool", "upsample", "shortcut", "route", "yolo", "avgpool", "softmax", "connected"};

constexpr unsigned long long STAGED_FROM = 2;   // steps on the driver's path for ordinary host memory, see upload
constexpr int MAX_PIECES = 8;   // parts the batch is cut into at most, see plan_step

// `count` images of the batch from `first` on; piece < 0 is the whole batch.
struct Part { int first, count, piece; };

// One unit of a step's schedule: layers begin .. end-1 over part of the batch, whose images are uploaded first where asked.
struct Item { int begin, end; Part part; bool uploads; };

struct Layer {
    LayerKind kind;
    int c, h, w;                   // input extents
    int out_c, out_h, out_w;
    dnb_tensor out;                // device output: NHWC in the network's storage type (yolo: NCHW f32)
    // convolutional; a connected layer is the 1x1 convolution of a 1x1 map whose channels are the whole input
    // (height x width x channel pitch of the channels-last tensor it reads), the batch folded into the pixel tile
    dnb_conv_desc cd;
    dnb_conv_plan *plan = nullptr;
    dnb_conv_plan *piece_plan[MAX_PIECES] = {};   // the same layer over one piece of the batch; the parameters are plan's
    bool flipped = false;          // convolutional: the file stores the weight matrix transposed (cfg flipped=1)
    int fc_inputs = 0;             // connected: inputs as the reference counts them (c*h*w of the previous layer)
    int in_cpitch = 0;             // connected: channel pitch of the tensor it reads
    // maxpool / upsample
    int size = 0, stride = 0, padding = 0;
    float scale = 1.f;
    // shortcut / route
    int from = -1;
    float alpha = 1.f, beta = 1.f;
    int activation = DNB_LINEAR;
    std::vector<int> inputs;
    // yolo
    int anchors = 0, classes = 0;
    float *host_out = nullptr;     // pinned; the slot of the step collected last
    float *host_slot[2] = {nullptr, nullptr};   // pinned result buffers of the two steps that may be in flight
    cudaEvent_t done = nullptr;    // compute stream: the layer's output is complete
    cudaEvent_t copied[MAX_PIECES] = {};   // copy stream: the device-to-host copy of a piece of that output is complete ([0]: of all of it, in one piece)
    bool params_given = false;     // dnb_network_set_conv_params has been called for this convolution
    // softmax
    int groups = 1;
    float temperature = 1.f;
    int launches = 1;
    // a convolution that also performs the [shortcut] layer right after it, and that shortcut layer
    bool fuses_next_shortcut = false, fused_into_prev = false;
    dnb_tensor own_out{};          // ... where that layer's addend has another shape: the convolution's own output, filled for who asks for it
    // a convolution that also performs the [yolo] layer right after it (that layer is then fused_into_prev too)
    bool fuses_next_yolo = false;
    // a convolution that also performs the 2x2 maxpool with stride 2 right after it (own_out is there for who asks for its own output)
    bool fuses_next_pool = false;
    // a maxpool layer that also writes the signs of its output, the next (tensor-core xnor) layer's operand
    int8_t *sign_out = nullptr;
    int sign_pitch = 0;
    // the output is a channel range of a later [route] layer's output: its producer writes it in place and the route
    // has nothing to copy for it (the memory belongs to the route layer)
    bool out_is_view = false;
};

typedef std::map<std::string, std::string> Options;

int opt_int(const Options &o, const char *k, int def)
{
    auto it = o.find(k);
    return it == o.end() ? def : atoi(it->second.c_str());
}
float opt_float(const Options &o, const char *k, float def)
{
    auto it = o.find(k);
    return it == o.end() ? def : (float)atof(it->second.c_str());
}
std::string opt_str(const Options &o, const char *k, const char *def)
{
    auto it = o.find(k);
    return it == o.end() ? std::string(def) : it->second;
}

// get_activation (src/activations.c:46-63): unknown names fall back to RELU there; here they are rejected.
int parse_activation(const std::string &s)
{
    static const char *const names[] = {"logistic", "relu", "relie", "linear", "ramp", "tanh", "plse",
                                        "leaky", "elu", "loggy", "stair", "hardtan", "lhtan", "selu"};
    for (int i = 0; i < 14; ++i)
        if (s == names[i]) return i;
    return -1;
}

std::string trim(const std::string &s)
{
    size_t a = s.find_first_not_of(" \t\r\n"), b = s.find_last_not_of(" \t\r\n");
    return a == std::string::npos ? std::string() : s.substr(a, b - a + 1);
}

// read_cfg (src/parser.c:891-924): '[' opens a section, '#' ';' and blank lines are skipped, the rest is key=value.
int split_cfg(const char *text, std::vector<std::pair<std::string, Options>> *sections)
{
    const char *p = text;
    int lineno = 0;
    while (*p) {
        const char *e = strchr(p, '\n');
        std::string line = trim(e ? std::string(p, e - p) : std::string(p));
        p = e ? e + 1 : p + strlen(p);
        ++lineno;
        if (line.empty() || line[0] == '#' || line[0] == ';') continue;
        if (line[0] == '[') {
            size_t r = line.find(']');
            if (r == std::string::npos) DNB_FAIL(DNB_EINVAL, "cfg line %d: unterminated section header", lineno);
            sections->push_back({trim(line.substr(1, r - 1)), Options()});
            continue;
        }
        size_t eq = line.find('=');
        if (eq == std::string::npos || sections->empty()) DNB_FAIL(DNB_EINVAL, "cfg line %d: expected key=value inside a section", lineno);
        sections->back().second[trim(line.substr(0, eq))] = trim(line.substr(eq + 1));
    }
    if (sections->empty()) DNB_FAIL(DNB_EINVAL, "cfg has no sections");
    return DNB_OK;
}

}  // namespace

struct dnb_network {
    int mode = DNB_MODE_TF32;
    int dtype = DNB_F32;             // storage type between layers
    int batch = 0, h = 0, w = 0, c = 0, inputs = 0, outputs = 0;
    std::vector<Layer> layers;
    float *input_dev = nullptr;      // NCHW f32 [batch][inputs]
    dnb_tensor input_nhwc{};         // only when the first layer needs channels-last input
    float *out_dev_nchw = nullptr;   // NCHW f32 staging of the output layer when it is not a yolo layer
    float *out_host = nullptr;       // pinned [batch][outputs]
    float *export_dev = nullptr;     // scratch for dnb_network_layer_output
    size_t export_elems = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t copy_stream = nullptr;   // device-to-host copies of finished [yolo] outputs, overlapping later layers
    cudaStream_t h2d_stream = nullptr;    // host-to-device copy of the next step's images
    float *input_slot[2] = {nullptr, nullptr};     // device images of the two steps that may be in flight ([0] is input_dev)
    float *out_host_slot[2] = {nullptr, nullptr};  // pinned output-layer results ([0] is out_host)
    cudaEvent_t in_ready[2] = {nullptr, nullptr}, fwd_done[2] = {nullptr, nullptr}, copy_done[2] = {nullptr, nullptr};
    unsigned long long submitted = 0, collected = 0;
    int *status_dev = nullptr;            // two time-out status words, one per step that may be in flight; every plan of
                                          // the network is pointed at the word of the step being enqueued
    int *status_host = nullptr;           // pinned copies, read when the step is collected
    int device = 0;
    bool weights_loaded = false;
    int convs_with_params = 0;
    // CUDA-graph replay of the device-resident forward (dnb_network_enable_graph): one instantiated graph per
    // (input pointer, stream) seen last; eager_runs counts forwards with that pair since it changed
    bool graph_enabled = false;
    cudaGraphExec_t graph_exec = nullptr;
    const float *graph_input = nullptr;
    cudaStream_t graph_stream = nullptr;
    int eager_runs = 0;
    std::vector<cudaEvent_t> events;
    // the blocking call replays its step, layers and result copies, as one graph per slot (see dnb_network_predict)
    cudaGraphExec_t step_exec[2] = {nullptr, nullptr};
    int step_runs[2] = {0, 0};
    bool step_graphs = true;              // off once something could not be captured
    const float *images = nullptr;        // the network's own buffer with the images of the last pass, where a first layer's own output is made on request
    std::vector<Item> schedule;           // a step, where its batch is enqueued in parts (see plan_step); else empty
    cudaEvent_t piece_in[MAX_PIECES] = {};   // upload stream: a piece's images are on the device
    std::vector<cudaGraphExec_t> item_exec[2];   // the schedule's items as graphs, per slot
    cudaEvent_t pulled = nullptr;         // copy stream: every result copy of a blocking step is enqueued
    std::shared_ptr<CopyPool> copier;     // held once an input in pageable memory asked for it
};

static void drop_graph(dnb_network *net);
static void plan_step(dnb_network *net);

static int alloc_activation(dnb_network *net, dnb_tensor *t, int c, int h, int w)
{
    t->layout = DNB_NHWC;
    t->dtype = net->dtype;
    t->n = net->batch; t->c = c; t->h = h; t->w = w;
    t->cpitch = round_up(c, 8);
    const size_t bytes = tensor_elems(t) * elem_size(t->dtype);
    DNB_CUDA(cudaMalloc(&t->data, bytes));
    DNB_CUDA(cudaMemset(t->data, 0, bytes));  // the cpitch - c padding channels stay zero for the lifetime of the network
    return DNB_OK;
}

static int build_network(const char *text, int mode, int batch_override, dnb_network **out)
{
    if (!text || !out) DNB_FAIL(DNB_EINVAL, "parse_network_cfg: null argument");
    *out = nullptr;
    if (mode != DNB_MODE_TF32 && mode != DNB_MODE_BF16 && mode != DNB_MODE_FP32) DNB_FAIL(DNB_EINVAL, "parse_network_cfg: mode %d", mode);
    std::vector<std::pair<std::string, Options>> sections;
    DNB_TRY(split_cfg(text, &sections));
    if (sections[0].first != "net" && sections[0].first != "network") DNB_FAIL(DNB_EINVAL, "cfg: first section must be [net] or [network]");

    dnb_network *net = new dnb_network();
    struct Guard { dnb_network *n; ~Guard() { if (n) dnb_free_network(n); } } guard{net};
    net->mode = mode;
    net->dtype = mode == DNB_MODE_BF16 ? DNB_BF16 : DNB_F32;
    DNB_CUDA(cudaGetDevice(&net->device));
    const Options &no = sections[0].second;
    // parse_net_options (src/parser.c:655-734): batch /= subdivisions
    int subdivs = opt_int(no, "subdivisions", 1);
    if (subdivs < 1) subdivs = 1;
    net->batch = batch_override > 0 ? batch_override : opt_int(no, "batch", 1) / subdivs;
    net->h = opt_int(no, "height", 0); net->w = opt_int(no, "width", 0); net->c = opt_int(no, "channels", 0);
    if (net->batch < 1 || net->h < 1 || net->w < 1 || net->c < 1)
        DNB_FAIL(DNB_EINVAL, "cfg [net]: need positive batch, height, width, channels (got %d, %d, %d, %d)", net->batch, net->h, net->w, net->c);
    net->inputs = net->h * net->w * net->c;

    int c = net->c, h = net->h, w = net->w;
    for (size_t si = 1; si < sections.size(); ++si) {
        const std::string &type = sections[si].first;
        const Options &o = sections[si].second;
        const int index = (int)si - 1;
        Layer L;
        L.c = c; L.h = h; L.w = w;
        if (type == "convolutional" || type == "conv") {
            L.kind = L_CONV;
            const int size = opt_int(o, "size", 1);
            int padding = opt_int(o, "padding", 0);
            if (opt_int(o, "pad", 0)) padding = size / 2;  // src/parser.c:184-187
            const int act = parse_activation(opt_str(o, "activation", "logistic"));
            if (act < 0) DNB_FAIL(DNB_EINVAL, "cfg layer %d: unknown activation '%s'", index, opt_str(o, "activation", "").c_str());
            L.cd = dnb_conv_desc{net->batch, h, w, c, opt_int(o, "filters", 1), opt_int(o, "groups", 1), size,
                                 opt_int(o, "stride", 1), padding, opt_int(o, "batch_normalize", 0), act, opt_int(o, "xnor", 0)};
            L.flipped = opt_int(o, "flipped", 0) != 0;   // parse_convolutional, src/parser.c:199: only the file's weight order differs
            DNB_TRY(dnb_conv_plan_create(&L.cd, mode, &L.plan));
            L.out_c = L.cd.n; L.out_h = L.plan->g.out_h; L.out_w = L.plan->g.out_w;
            L.launches = L.plan->kernel == 3 ? 2 : 1;
        } else if (type == "connected" || type == "conn") {
            // parse_connected (src/parser.c:259-268), make_connected_layer (src/connected_layer.c:14-33)
            L.kind = L_CONNECTED;
            const int act = parse_activation(opt_str(o, "activation", "logistic"));
            if (act < 0) DNB_FAIL(DNB_EINVAL, "cfg layer %d: unknown activation '%s'", index, opt_str(o, "activation", "").c_str());
            const int outputs = opt_int(o, "output", 1);
            if (outputs < 1) DNB_FAIL(DNB_EINVAL, "cfg layer %d: connected output=%d", index, outputs);
            L.fc_inputs = c * h * w;
            L.in_cpitch = round_up(c, 8);
            L.cd = dnb_conv_desc{net->batch, 1, 1, h * w * L.in_cpitch, outputs, 1, 1, 1, 0, opt_int(o, "batch_normalize", 0), act, 0};
            DNB_TRY(dnb_conv_plan_create(&L.cd, mode, &L.plan));
            L.out_c = outputs; L.out_h = 1; L.out_w = 1;
        } else if (type == "maxpool" || type == "max") {
            L.kind = L_MAXPOOL;
            L.stride = opt_int(o, "stride", 1);
            L.size = opt_int(o, "size", L.stride);
            L.padding = opt_int(o, "padding", L.size - 1);  // src/parser.c:485-487
            if (L.stride < 1 || L.size < 1) DNB_FAIL(DNB_EINVAL, "cfg layer %d: maxpool size %d stride %d", index, L.size, L.stride);
            L.out_c = c; L.out_h = (h + L.padding - L.size) / L.stride + 1; L.out_w = (w + L.padding - L.size) / L.stride + 1;
        } else if (type == "upsample") {
            L.kind = L_UPSAMPLE;
            L.stride = opt_int(o, "stride", 2);
            L.scale = opt_float(o, "scale", 1.f);
            if (L.stride < 1) DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: upsample stride %d (reverse form)", index, L.stride);
            L.out_c = c; L.out_h = h * L.stride; L.out_w = w * L.stride;
        } else if (type == "shortcut") {
            L.kind = L_SHORTCUT;
            int from = opt_int(o, "from", 0);
            if (o.find("from") == o.end()) DNB_FAIL(DNB_EINVAL, "cfg layer %d: shortcut without from=", index);
            if (from < 0) from = index + from;
            if (from < 0 || from >= index) DNB_FAIL(DNB_EINVAL, "cfg layer %d: shortcut from=%d out of range", index, from);
            L.from = from;
            L.activation = parse_activation(opt_str(o, "activation", "linear"));
            if (L.activation < 0) DNB_FAIL(DNB_EINVAL, "cfg layer %d: unknown activation", index);
            L.alpha = opt_float(o, "alpha", 1.f); L.beta = opt_float(o, "beta", 1.f);
            L.out_c = c; L.out_h = h; L.out_w = w;
        } else if (type == "route") {
            L.kind = L_ROUTE;
            std::string ls = opt_str(o, "layers", "");
            if (ls.empty()) DNB_FAIL(DNB_EINVAL, "cfg layer %d: route must specify input layers", index);
            size_t pos = 0;
            int csum = 0;
            while (pos <= ls.size()) {
                size_t comma = ls.find(',', pos);
                int id = atoi(ls.substr(pos, comma == std::string::npos ? std::string::npos : comma - pos).c_str());
                if (id < 0) id = index + id;
                if (id < 0 || id >= index) DNB_FAIL(DNB_EINVAL, "cfg layer %d: route input %d out of range", index, id);
                L.inputs.push_back(id);
                csum += net->layers[id].out_c;
                if (comma == std::string::npos) break;
                pos = comma + 1;
            }
            const Layer &first = net->layers[L.inputs[0]];
            for (int id : L.inputs)
                if (net->layers[id].out_h != first.out_h || net->layers[id].out_w != first.out_w)
                    DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: route inputs of unequal width/height", index);
            L.out_c = csum; L.out_h = first.out_h; L.out_w = first.out_w;
            L.launches = (int)L.inputs.size();
        } else if (type == "yolo") {
            L.kind = L_YOLO;
            // parse_yolo (src/parser.c:306-345): n = number of mask entries (or num), classes default 20
            const std::string mask = opt_str(o, "mask", "");
            int n = opt_int(o, "num", 1);
            if (!mask.empty()) { n = 1; for (char ch : mask) if (ch == ',') ++n; }
            L.anchors = n; L.classes = opt_int(o, "classes", 20);
            if (c != n * (L.classes + 5)) DNB_FAIL(DNB_EINVAL, "cfg layer %d: yolo expects %d channels, input has %d", index, n * (L.classes + 5), c);
            L.out_c = c; L.out_h = h; L.out_w = w;
        } else if (type == "avgpool" || type == "avg") {
            L.kind = L_AVGPOOL;
            L.out_c = c; L.out_h = 1; L.out_w = 1;
        } else if (type == "softmax" || type == "soft") {
            L.kind = L_SOFTMAX;
            L.groups = opt_int(o, "groups", 1);
            L.temperature = opt_float(o, "temperature", 1.f);
            if (o.find("tree") != o.end()) DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: softmax tree", index);
            if (h != 1 || w != 1) DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: softmax over a %dx%d map", index, w, h);
            L.out_c = c; L.out_h = 1; L.out_w = 1;
        } else {
            DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: section [%s] is outside the convolutional forward path", index, type.c_str());
        }
        if (L.out_h < 1 || L.out_w < 1) DNB_FAIL(DNB_EINVAL, "cfg layer %d: empty output", index);
        // the previous layer's output must be channels-last for every consumer but none reads a yolo output
        if (index > 0 && net->layers[index - 1].kind == L_YOLO && L.kind != L_ROUTE)
            DNB_FAIL(DNB_EUNSUPPORTED, "cfg layer %d: a [%s] directly after [yolo]", index, type.c_str());
        if (L.kind == L_YOLO) {
            L.out = dnb_tensor{nullptr, DNB_NCHW, DNB_F32, net->batch, L.out_c, L.out_h, L.out_w, 0};
            const size_t bytes = tensor_elems(&L.out) * sizeof(float);
            DNB_CUDA(cudaMalloc(&L.out.data, bytes));
            DNB_CUDA(cudaMallocHost((void **)&L.host_slot[0], bytes));
            L.host_out = L.host_slot[0];
        } else {
            DNB_TRY(alloc_activation(net, &L.out, L.out_c, L.out_h, L.out_w));
        }
        net->layers.push_back(L);
        c = L.out_c; h = L.out_h; w = L.out_w;
    }
    if (net->layers.empty()) DNB_FAIL(DNB_EINVAL, "cfg has no layers");
    for (const Layer &L : net->layers) {
        if (L.kind == L_SHORTCUT && net->layers[L.from].kind == L_YOLO) DNB_FAIL(DNB_EUNSUPPORTED, "cfg: shortcut from a [yolo] layer");
        if (L.kind == L_ROUTE)
            for (int id : L.inputs)
                if (net->layers[id].kind == L_YOLO) DNB_FAIL(DNB_EUNSUPPORTED, "cfg: route from a [yolo] layer");
    }
    bool any_xnor = false;
    for (const Layer &L : net->layers) any_xnor = any_xnor || (L.kind == L_CONV && L.cd.xnor);
    // Fuse "convolution, then [shortcut]" (of equal shape, or as ResNet's stages begin: fewer channels, a larger map) into
    // the convolution's epilogue when nothing else reads the convolution's own output: one pass over the activations
    // instead of three.  (ResNet-50, batch 256: the four passes that had other shapes took 0.86 ms of 7.7.)
    // DNB_FUSE_SHORTCUT=0 keeps every layer separate (every layer's output stays readable).
    const bool fuse = getenv("DNB_FUSE_SHORTCUT") ? atoi(getenv("DNB_FUSE_SHORTCUT")) != 0 : true;
    for (int i = 0; fuse && i + 1 < (int)net->layers.size(); ++i) {
        Layer &C = net->layers[i], &S = net->layers[i + 1];
        if (C.kind != L_CONV || !C.plan || (C.plan->kernel != 0 && C.plan->kernel != 1) || S.kind != L_SHORTCUT || S.from == i) continue;
        const Layer &F = net->layers[S.from];
        if (F.kind == L_YOLO || !conv_shortcut_fusable(C.plan, &F.out, &S.out, S.alpha)) continue;
        const bool other_shape = F.out.c != S.out.c || F.out.h != S.out.h || F.out.w != S.out.w;
        if (other_shape && any_xnor) continue;   // their sums, which layers take the signs of, are rounded where they always were
        bool read_elsewhere = false;
        for (int j = i + 2; j < (int)net->layers.size(); ++j) {
            const Layer &L = net->layers[j];
            if (L.kind == L_SHORTCUT && L.from == i) read_elsewhere = true;
            if (L.kind == L_ROUTE)
                for (int id : L.inputs) if (id == i) read_elsewhere = true;
        }
        if (read_elsewhere) continue;
        C.fuses_next_shortcut = true;
        S.fused_into_prev = true;
        S.launches = 0;
        // Never written by a step: the convolution stores straight into the shortcut's output.  An output that was to be read while
        // only equal shapes were fused still is (own_output).
        if (other_shape) C.own_out = C.out;
        else cudaFree(C.out.data);
        C.out.data = nullptr;
    }
    // Fuse "convolution, then [yolo]" when nothing else reads the convolution's output: the epilogue applies the yolo
    // layer's logistic per entry and writes that layer's NCHW output; the channels-last copy of the raw predictions
    // and the pass that transposed it (forward_yolo_layer_gpu, src/yolo_layer.c:347-357) disappear.
    // DNB_FUSE_YOLO=0 keeps the two layers separate.
    const bool fuse_yolo = getenv("DNB_FUSE_YOLO") ? atoi(getenv("DNB_FUSE_YOLO")) != 0 : true;
    for (int i = 0; fuse_yolo && i + 1 < (int)net->layers.size(); ++i) {
        Layer &C = net->layers[i], &Y = net->layers[i + 1];
        if (C.kind != L_CONV || !C.plan || (C.plan->kernel != 0 && C.plan->kernel != 1) || C.plan->stem_tc || Y.kind != L_YOLO) continue;
        if (C.plan->d.activation != DNB_LINEAR || C.plan->g.n % 256 == 0) continue;   // the fused epilogue is built for the linear heads every yolo cfg has (and not for CTA pairs)
        bool read_elsewhere = false;
        for (int j = i + 2; j < (int)net->layers.size(); ++j) {
            const Layer &L = net->layers[j];
            if (L.kind == L_SHORTCUT && L.from == i) read_elsewhere = true;
            if (L.kind == L_ROUTE)
                for (int id : L.inputs) if (id == i) read_elsewhere = true;
        }
        if (read_elsewhere) continue;
        C.fuses_next_yolo = true;
        Y.fused_into_prev = true;
        Y.launches = 0;
        cudaFree(C.out.data);      // never written: the convolution stores straight into the yolo layer's output
        C.out.data = nullptr;
    }
    // Fuse "convolution, then 2x2 [maxpool] with stride 2" when nothing else reads the convolution's output: its epilogue writes the largest of
    // each four pixels, and the pass that read the whole map back disappears.  The convolution's own output is made from its input for
    // who asks for it (own_output).  DNB_FUSE_POOL=0 keeps the two layers separate.
    const bool fuse_pool = getenv("DNB_FUSE_POOL") ? atoi(getenv("DNB_FUSE_POOL")) != 0 : true;
    for (int i = 0; i + 1 < (int)net->layers.size(); ++i) {
        Layer &C = net->layers[i], &M = net->layers[i + 1];
        if (C.kind != L_CONV || !C.plan || M.kind != L_MAXPOOL || M.size != 2 || M.stride != 2 || M.padding < 0 || M.padding > 1 || !C.out.data) continue;
        if (M.out_h != C.out_h / 2 || M.out_w != C.out_w / 2) continue;
        bool read_elsewhere = false, sign_pass = false;
        for (int j = i + 2; j < (int)net->layers.size(); ++j) {
            const Layer &L = net->layers[j];
            if (L.kind == L_SHORTCUT && L.from == i) read_elsewhere = true;
            if (L.kind == L_ROUTE)
                for (int id : L.inputs) if (id == i) read_elsewhere = true;
            // the maxpool kernel also writes the next xnor layer's operand; of the convolutions only an xnor layer or a first one does
            if (j == i + 2 && L.kind == L_CONV && L.cd.xnor && !C.cd.xnor && !C.plan->stem_tc) sign_pass = true;
        }
        if (read_elsewhere || sign_pass || !conv_pool_fusable(C.plan, any_xnor)) continue;
        if (i == 0 && net->mode == DNB_MODE_BF16 && C.out.dtype != DNB_BF16) continue;
        C.plan->tap_order = true;   // the same sums whether the two layers are one launch or two
        if (!fuse_pool) continue;
        C.fuses_next_pool = true;
        M.fused_into_prev = true;
        M.launches = 0;
        C.own_out = C.out;
        C.out.data = nullptr;
    }
    // Zero-copy [route]: where a route input is produced by a layer whose kernel can write a channel range of a wider
    // channels-last tensor (tensor-core convolutions, with or without a fused shortcut, and upsample), and everything that
    // reads it can read such a range (convolutions, routes, the yolo head, upsample), the input's tensor BECOMES its
    // range of the route's output: forward_route_layer_gpu's copies (src/route_layer.c:105-118) disappear.
    // DNB_ROUTE_ALIAS=0 keeps every layer's own tensor.
    const bool alias = getenv("DNB_ROUTE_ALIAS") ? atoi(getenv("DNB_ROUTE_ALIAS")) != 0 : true;
    for (int r = 0; alias && r < (int)net->layers.size(); ++r) {
        Layer &R = net->layers[r];
        if (R.kind != L_ROUTE) continue;
        const size_t es = elem_size(R.out.dtype);
        int off = 0, copies = 0;
        for (size_t k = 0; k < R.inputs.size(); ++k) {
            const int id = R.inputs[k];
            Layer &P = net->layers[id];
            const int this_off = off;
            off += P.out_c;
            ++copies;
            const bool last_input = k + 1 == R.inputs.size();
            if (P.out_is_view || !P.out.data || P.out.layout != DNB_NHWC) continue;
            if ((size_t)this_off * es % 128 || (!last_input && P.out_c % 8)) continue;
            bool writer_ok = false;
            if (P.kind == L_UPSAMPLE) writer_ok = true;
            if (P.kind == L_CONV && P.plan && (P.plan->kernel == 0 || P.plan->kernel == 1) && !P.plan->stem_tc) writer_ok = true;
            if (P.kind == L_SHORTCUT && P.fused_into_prev) writer_ok = true;   // written by the convolution before it
            if (!writer_ok) continue;
            bool readers_ok = true;
            for (int j = id + 1; j < (int)net->layers.size() && readers_ok; ++j) {
                const Layer &C = net->layers[j];
                const bool reads_as_input = j == id + 1 && C.kind != L_ROUTE && !(C.kind == L_SHORTCUT && C.fused_into_prev);
                if (reads_as_input && !(C.kind == L_CONV && !C.plan->stem_tc) && C.kind != L_YOLO && C.kind != L_UPSAMPLE) readers_ok = false;
                if (C.kind == L_SHORTCUT && C.from == id && !C.fused_into_prev) readers_ok = false;   // the stand-alone kernel wants equal pitches
            }
            if (!readers_ok) continue;
            cudaFree(P.out.data);
            P.out.data = (char *)R.out.data + (size_t)this_off * es;
            P.out.cpitch = R.out.cpitch;
            P.out_is_view = true;
            --copies;
        }
        R.launches = copies;
    }
    // xnor layers in a row: the first one's epilogue writes the second one's int8 operand (conv_plan_link_signs)
    for (int i = 0; i + 1 < (int)net->layers.size(); ++i) {
        Layer &A = net->layers[i], &B = net->layers[i + 1];
        if (B.kind != L_CONV || !B.plan || !A.out.data || A.out.layout != DNB_NHWC) continue;
        if (A.kind == L_CONV && A.plan) {
            if (conv_plan_link_signs(A.plan, B.plan, A.out.data)) B.launches = 1;   // no sign pass of its own
        } else if (A.kind == L_MAXPOOL && A.fused_into_prev) {
            if (conv_plan_link_signs(net->layers[i - 1].plan, B.plan, A.out.data, true)) B.launches = 1;
        } else if (A.kind == L_MAXPOOL && A.out.dtype == DNB_F32 && A.out.cpitch == A.out_c) {
            A.sign_out = conv_plan_expect_signs(B.plan, A.out.data, net->batch, A.out_c, A.out_h, A.out_w);
            if (A.sign_out) { A.sign_pitch = A.out_c; B.launches = 1; }
        }
    }
    // A sign hangs on a sum's last bit.  Where layers are binarised, the dense ones add in the same order at every batch
    // size (integer sums do not care), so that an image's results do not depend on how many came with it, and a first layer
    // on the tensor cores adds in the reference's order of the products.
    for (Layer &L : net->layers) if (L.plan) L.plan->keep_k_order = any_xnor;
    // Sums stay in one order where their last bits grow: a classifier's [softmax] makes 0.015 of a probability of one TF32 bit (ResNet-50, 256 images), and
    // bf16 roundings add up over a network's layers (YOLOv3's outputs move by 1 to 2 % with the order, those of YOLOv3-tiny by 0.25).
    bool any_softmax = false;
    for (const Layer &L : net->layers) any_softmax |= L.kind == L_SOFTMAX;
    if (any_softmax || net->mode == DNB_MODE_BF16)
        for (Layer &L : net->layers) if (L.plan) L.plan->tap_order = true;
    const Layer &last = net->layers.back();
    net->outputs = last.out_c * last.out_h * last.out_w;
    DNB_CUDA(cudaMalloc((void **)&net->input_dev, (size_t)net->batch * net->inputs * sizeof(float)));
    DNB_CUDA(cudaMallocHost((void **)&net->out_host, (size_t)net->batch * net->outputs * sizeof(float)));
    if (last.kind != L_YOLO) DNB_CUDA(cudaMalloc((void **)&net->out_dev_nchw, (size_t)net->batch * net->outputs * sizeof(float)));
    const Layer &first = net->layers.front();
    const bool first_reads_nchw = first.kind == L_CONV && (first.plan->kernel == 2 || first.plan->kernel == 3);   // a connected first layer reads the channels-last copy
    if (!first_reads_nchw) {
        dnb_tensor *t = &net->input_nhwc;
        DNB_TRY(alloc_activation(net, t, net->c, net->h, net->w));
    }
    DNB_CUDA(cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking));
    DNB_CUDA(cudaStreamCreateWithFlags(&net->copy_stream, cudaStreamNonBlocking));
    DNB_CUDA(cudaStreamCreateWithFlags(&net->h2d_stream, cudaStreamNonBlocking));
    net->input_slot[0] = net->input_dev;
    net->out_host_slot[0] = net->out_host;
    for (int k = 0; k < 2; ++k) {
        DNB_CUDA(cudaEventCreateWithFlags(&net->in_ready[k], cudaEventDisableTiming));
        DNB_CUDA(cudaEventCreateWithFlags(&net->fwd_done[k], cudaEventDisableTiming));
        DNB_CUDA(cudaEventCreateWithFlags(&net->copy_done[k], cudaEventDisableTiming));
    }
    for (Layer &L : net->layers)
        if (L.kind == L_YOLO) {
            DNB_CUDA(cudaEventCreateWithFlags(&L.done, cudaEventDisableTiming));
            for (cudaEvent_t &e : L.copied) DNB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        }
    DNB_CUDA(cudaEventCreateWithFlags(&net->pulled, cudaEventDisableTiming));
    for (cudaEvent_t &e : net->piece_in) DNB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    plan_step(net);
    DNB_CUDA(cudaMalloc((void **)&net->status_dev, 2 * sizeof(int)));
    DNB_CUDA(cudaMemset(net->status_dev, 0, 2 * sizeof(int)));
    DNB_CUDA(cudaMallocHost((void **)&net->status_host, 2 * sizeof(int)));
    net->status_host[0] = net->status_host[1] = 0;
    for (Layer &L : net->layers)
        if (L.plan) { L.plan->status = net->status_dev; L.plan->status_shared = true; }
    guard.n = nullptr;
    *out = net;
    return DNB_OK;
}

extern "C" int dnb_parse_network_cfg_text(const char *cfg_text, int mode, int batch_override, dnb_network **net)
{
    return build_network(cfg_text, mode, batch_override, net);
}

extern "C" int dnb_parse_network_cfg(const char *path, int mode, int batch_override, dnb_network **net)
{
    if (!path) DNB_FAIL(DNB_EINVAL, "parse_network_cfg: null path");
    FILE *f = fopen(path, "rb");
    if (!f) DNB_FAIL(DNB_EIO, "Couldn't open file: %s", path);  // file_error, src/utils.c:281-285
    std::string text;
    char buf[4096];
    size_t n;
    while ((n = fread(buf, 1, sizeof(buf), f)) > 0) text.append(buf, n);
    fclose(f);
    return build_network(text.c_str(), mode, batch_override, net);
}

extern "C" void dnb_free_network(dnb_network *net)
{
    if (!net) return;
    drop_graph(net);
    for (Layer &L : net->layers) {
        if (L.plan) dnb_conv_plan_destroy(L.plan);
        if (!L.out_is_view) cudaFree(L.out.data);
        cudaFree(L.own_out.data);
        for (float *hp : L.host_slot) if (hp) cudaFreeHost(hp);
        for (cudaEvent_t e : L.copied) if (e) cudaEventDestroy(e);
    }
    cudaFree(net->input_dev); cudaFree(net->input_nhwc.data); cudaFree(net->out_dev_nchw); cudaFree(net->export_dev);
    if (net->out_host) cudaFreeHost(net->out_host);
    if (net->status_host) cudaFreeHost(net->status_host);
    for (cudaEvent_t e : net->piece_in) if (e) cudaEventDestroy(e);
    if (net->pulled) cudaEventDestroy(net->pulled);
    cudaFree(net->status_dev);
    for (cudaEvent_t e : net->events) cudaEventDestroy(e);
    for (Layer &L : net->layers) if (L.done) cudaEventDestroy(L.done);
    if (net->stream) cudaStreamDestroy(net->stream);
    if (net->copy_stream) cudaStreamDestroy(net->copy_stream);
    if (net->h2d_stream) cudaStreamDestroy(net->h2d_stream);
    cudaFree(net->input_slot[1]);
    if (net->out_host_slot[1]) cudaFreeHost(net->out_host_slot[1]);
    for (int k = 0; k < 2; ++k) {
        if (net->in_ready[k]) cudaEventDestroy(net->in_ready[k]);
        if (net->fwd_done[k]) cudaEventDestroy(net->fwd_done[k]);
        if (net->copy_done[k]) cudaEventDestroy(net->copy_done[k]);
    }
    delete net;
}

// A connected layer's matrix, [outputs][inputs] with the inputs in the reference's order (channel, row, column of the
// previous layer's output, src/connected_layer.c:151-160), rearranged for the channels-last tensor the layer reads
// here: input (ch, y, x) sits at ((y * w + x) * cpitch + ch); padding channels get zero weights.
static int set_connected_params(dnb_network *net, Layer &L, int index, const float *weights, const float *biases, const float *scales,
                                const float *mean, const float *var)
{
    const Layer *prev = index > 0 ? &net->layers[index - 1] : nullptr;
    const int c = prev ? prev->out_c : net->c, h = prev ? prev->out_h : net->h, w = prev ? prev->out_w : net->w;
    const int cp = L.in_cpitch, outputs = L.cd.n;
    const size_t k = (size_t)h * w * cp;
    std::vector<float> packed((size_t)outputs * k, 0.f);
    for (int o = 0; o < outputs; ++o)
        for (int ch = 0; ch < c; ++ch)
            for (int y = 0; y < h; ++y)
                for (int x = 0; x < w; ++x)
                    packed[(size_t)o * k + ((size_t)y * w + x) * cp + ch] = weights[(size_t)o * L.fc_inputs + ((size_t)ch * h + y) * w + x];
    return dnb_conv_plan_set_params(L.plan, packed.data(), biases, scales, mean, var);
}

// Before the first parameter tensor is replaced: no step of the network is under way, and nothing that holds the tensors' pointers
// (captured steps, the plans of parts of a batch) is left, however the replacing ends.
static int release_params(dnb_network *net)
{
    DNB_TRY(check_current_device(net->device, "network parameters"));
    DNB_CUDA(cudaStreamSynchronize(net->h2d_stream));
    DNB_CUDA(cudaStreamSynchronize(net->stream));
    DNB_CUDA(cudaStreamSynchronize(net->copy_stream));
    drop_graph(net);
    return DNB_OK;
}

// ... of all layers: the network predicts again once every one of them has new parameters.
static int begin_params(dnb_network *net)
{
    DNB_TRY(release_params(net));
    net->weights_loaded = false;
    net->convs_with_params = 0;
    for (Layer &L : net->layers) L.params_given = false;
    return DNB_OK;
}

static int load_weights_impl(dnb_network *net, const char *path, bool packed)
{
    if (!net || !path) DNB_FAIL(DNB_EINVAL, "load_weights: null argument");
    FILE *f = fopen(path, "rb");
    if (!f) DNB_FAIL(DNB_EIO, "Couldn't open file: %s", path);
    struct Closer { FILE *f; ~Closer() { fclose(f); } } closer{f};
    int hdr[3];
    if (fread(hdr, sizeof(int), 3, f) != 3) DNB_FAIL(DNB_EIO, "%s: truncated header", path);
    // src/parser.c:1234-1241: a 64-bit `seen` from version 0.2 on, a 32-bit one before
    if ((hdr[0] * 10 + hdr[1]) >= 2 && hdr[0] < 1000 && hdr[1] < 1000) {
        uint64_t seen;
        if (fread(&seen, sizeof(seen), 1, f) != 1) DNB_FAIL(DNB_EIO, "%s: truncated header", path);
    } else {
        int seen;
        if (fread(&seen, sizeof(seen), 1, f) != 1) DNB_FAIL(DNB_EIO, "%s: truncated header", path);
    }
    // File versions above 1000 store connected-layer matrices as [inputs][outputs] (src/parser.c:1244, 1098-1104);
    // convolutional layers are not affected by the version.
    const bool transposed = hdr[0] > 1000 || hdr[1] > 1000;
    DNB_TRY(begin_params(net));
    int index = 0;
    for (Layer &L : net->layers) {
        if (L.kind == L_CONV) {
            // load_convolutional_weights (src/parser.c:1164-1215): biases, batchnorm vectors, weights
            const dnb_conv_desc &d = L.cd;
            const size_t nw = (size_t)d.n * (d.c / d.groups) * d.size * d.size;
            std::vector<float> biases(d.n), scales, mean, var, weights(nw);
            bool ok = fread(biases.data(), sizeof(float), d.n, f) == (size_t)d.n;
            if (ok && d.batch_normalize) {
                scales.resize(d.n); mean.resize(d.n); var.resize(d.n);
                ok = fread(scales.data(), sizeof(float), d.n, f) == (size_t)d.n &&
                     fread(mean.data(), sizeof(float), d.n, f) == (size_t)d.n &&
                     fread(var.data(), sizeof(float), d.n, f) == (size_t)d.n;
            }
            if (ok && packed && d.xnor) {
                // load_convolutional_weights_binary (src/parser.c:1134-1162): per filter its mean |w| as a float, then one
                // bit per weight (set: +mean, clear: -mean), eight to a byte, lowest bit first.  The reference stores
                // size/8 bytes per filter, so a filter whose c*size*size is not a multiple of 8 would lose its tail.
                const size_t per = nw / d.n;
                if (per % 8) DNB_FAIL(DNB_EUNSUPPORTED, "%s: layer %d has %zu weights per filter; the packed format holds whole bytes of 8 only", path, index, per);
                std::vector<unsigned char> bits(per / 8);
                for (int n = 0; n < d.n && ok; ++n) {
                    float mean = 0;
                    ok = fread(&mean, sizeof(float), 1, f) == 1 && fread(bits.data(), 1, per / 8, f) == per / 8;
                    for (size_t k = 0; ok && k < per; ++k) weights[(size_t)n * per + k] = (bits[k / 8] >> (k % 8)) & 1 ? mean : -mean;
                }
            } else {
                ok = ok && fread(weights.data(), sizeof(float), nw, f) == nw;
            }
            if (!ok) DNB_FAIL(DNB_EIO, "%s: file ends inside layer %d (the reference would silently keep its random initialisation)", path, index);
            if (L.flipped) {
                // transpose_matrix(l.weights, l.c*l.size*l.size, l.n) (src/parser.c:1206-1208, 1085-1096): the file holds
                // c*size*size rows of n values; Darknet's layout is n rows of c*size*size values
                const size_t rows = nw / d.n, cols = d.n;
                std::vector<float> t(nw);
                for (size_t x = 0; x < rows; ++x)
                    for (size_t y = 0; y < cols; ++y) t[y * rows + x] = weights[x * cols + y];
                weights.swap(t);
            }
            DNB_TRY(dnb_conv_plan_set_params(L.plan, weights.data(), biases.data(), d.batch_normalize ? scales.data() : nullptr,
                                             d.batch_normalize ? mean.data() : nullptr, d.batch_normalize ? var.data() : nullptr));
        } else if (L.kind == L_CONNECTED) {
            // load_connected_weights (src/parser.c:1098-1120): biases, weights, then the batchnorm vectors
            const int outputs = L.cd.n, inputs = L.fc_inputs;
            const size_t nw = (size_t)outputs * inputs;
            std::vector<float> biases(outputs), scales, mean, var, weights(nw);
            bool ok = fread(biases.data(), sizeof(float), outputs, f) == (size_t)outputs && fread(weights.data(), sizeof(float), nw, f) == nw;
            if (ok && L.cd.batch_normalize) {
                scales.resize(outputs); mean.resize(outputs); var.resize(outputs);
                ok = fread(scales.data(), sizeof(float), outputs, f) == (size_t)outputs &&
                     fread(mean.data(), sizeof(float), outputs, f) == (size_t)outputs &&
                     fread(var.data(), sizeof(float), outputs, f) == (size_t)outputs;
            }
            if (!ok) DNB_FAIL(DNB_EIO, "%s: file ends inside layer %d", path, index);
            if (transposed) {
                std::vector<float> t(nw);   // transpose_matrix(l.weights, l.inputs, l.outputs)
                for (int x = 0; x < inputs; ++x)
                    for (int y = 0; y < outputs; ++y) t[(size_t)y * inputs + x] = weights[(size_t)x * outputs + y];
                weights.swap(t);
            }
            DNB_TRY(set_connected_params(net, L, index, weights.data(), biases.data(), L.cd.batch_normalize ? scales.data() : nullptr,
                                         L.cd.batch_normalize ? mean.data() : nullptr, L.cd.batch_normalize ? var.data() : nullptr));
        }
        ++index;
    }
    net->weights_loaded = true;
    return DNB_OK;
}

extern "C" int dnb_load_weights(dnb_network *net, const char *path) { return load_weights_impl(net, path, false); }

// The same file format with every xnor convolution stored packed (mean |w| and one sign bit per weight).
extern "C" int dnb_load_weights_packed(dnb_network *net, const char *path) { return load_weights_impl(net, path, true); }

// The same derived tensors from host arrays instead of a file: what a host that has already run the
// reference's load_weights holds in l.weights, l.biases, l.scales, l.rolling_mean, l.rolling_variance.
extern "C" int dnb_network_set_conv_params(dnb_network *net, int layer, const float *weights, const float *biases,
                                           const float *scales, const float *rolling_mean, const float *rolling_variance)
{
    if (!net || layer < 0 || layer >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "set_conv_params: bad argument");
    Layer &L = net->layers[layer];
    if (L.kind != L_CONV && L.kind != L_CONNECTED) DNB_FAIL(DNB_EINVAL, "set_conv_params: layer %d has no parameters", layer);
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "set_conv_params: a submitted step is still in flight; collect it first");
    DNB_TRY(release_params(net));
    if (L.kind == L_CONNECTED) {
        if (!weights || !biases) DNB_FAIL(DNB_EINVAL, "set_conv_params: null argument");
        DNB_TRY(set_connected_params(net, L, layer, weights, biases, scales, rolling_mean, rolling_variance));
    } else {
        DNB_TRY(dnb_conv_plan_set_params(L.plan, weights, biases, scales, rolling_mean, rolling_variance));
    }
    if (!L.params_given) { L.params_given = true; ++net->convs_with_params; }
    int convs = 0;
    for (const Layer &K : net->layers) convs += K.kind == L_CONV || K.kind == L_CONNECTED;
    if (net->convs_with_params == convs) net->weights_loaded = true;
    return DNB_OK;
}

// Layer i's output as a step leaves it, in *t; the own output of a convolution that was fused with a shortcut of another shape or a maxpool is
// made from its input, which is still there, on s.
static int own_output(dnb_network *net, int i, dnb_tensor *t, cudaStream_t s)
{
    Layer &L = net->layers[i];
    *t = L.out;
    if (L.out.data) return DNB_OK;
    if (!L.own_out.data)
        DNB_FAIL(DNB_EUNSUPPORTED, "layer %d is fused into layer %d and has no output of its own (DNB_FUSE_SHORTCUT=0 / DNB_FUSE_YOLO=0 keep it)", i, i + 1);
    if (i == 0 && !net->input_nhwc.data && !net->images) DNB_FAIL(DNB_EINVAL, "layer 0: no step has run");
    const dnb_tensor in = i > 0 ? net->layers[i - 1].out : net->input_nhwc.data ? net->input_nhwc
                          : dnb_tensor{(void *)net->images, DNB_NCHW, DNB_F32, net->batch, net->c, net->h, net->w, 0};
    *t = L.own_out;
    return dnb_conv_forward(L.plan, &in, t, nullptr, s);
}

// Layer `layer`'s current output in Darknet's layout (NCHW f32) into device memory of the caller, on `stream`.
extern "C" int dnb_network_export_layer(dnb_network *net, int layer, float *device_nchw, void *stream)
{
    if (!net || !device_nchw || layer < 0 || layer >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "export_layer: bad argument");
    Layer &L = net->layers[layer];
    cudaStream_t s = (cudaStream_t)stream;
    dnb_tensor out;
    DNB_TRY(own_output(net, layer, &out, s));
    if (L.out.layout == DNB_NCHW) {
        DNB_CUDA(cudaMemcpyAsync(device_nchw, L.out.data, tensor_elems(&L.out) * sizeof(float), cudaMemcpyDeviceToDevice, s));
        return DNB_OK;
    }
    dnb_tensor o{device_nchw, DNB_NCHW, DNB_F32, net->batch, L.out_c, L.out_h, L.out_w, 0};
    return launch_convert(&out, &o, 0, 0, 0, s);
}

// Every convolution launched from here on reports an expired wait in the status word of step slot `slot`.
static void point_status(dnb_network *net, int slot)
{
    for (Layer &L : net->layers)
        if (L.plan) {
            L.plan->status = net->status_dev + slot;
            for (dnb_conv_plan *q : L.piece_plan) if (q) q->status = L.plan->status;
        }
}

static const char *const kTimeoutText =
    "a device-side wait expired in a convolution (code %d: 101 ring slot free, 102 operands landed, 103 accumulator free, "
    "104 accumulator ready, 105 residual tile, 106 shared memory window not 1024-byte aligned); the outputs are incomplete";

static Part whole(const dnb_network *net) { return Part{0, net->batch, -1}; }

static dnb_tensor part_of(const dnb_tensor &t, const Part &p)
{
    dnb_tensor r = t;
    if (p.piece < 0 || !t.data) return r;
    r.data = (char *)t.data + tensor_elems(&t) / t.n * p.first * elem_size(t.dtype);
    r.n = p.count;
    return r;
}

static dnb_conv_plan *plan_of(Layer &L, const Part &p)
{
    if (p.piece < 0) return L.plan;
    if (!L.piece_plan[p.piece]) L.piece_plan[p.piece] = conv_plan_for_batch(L.plan, p.count);
    return L.piece_plan[p.piece];
}

// Transposes the network input into channels-last form when the first layer wants that.
static int prepare_input(dnb_network *net, const float *device_input, const Part &p, cudaStream_t s)
{
    if (!net->input_nhwc.data) return DNB_OK;
    const dnb_tensor in = part_of(dnb_tensor{(void *)device_input, DNB_NCHW, DNB_F32, net->batch, net->c, net->h, net->w, 0}, p), out = part_of(net->input_nhwc, p);
    return launch_convert(&in, &out, net->mode == DNB_MODE_TF32, 0, 0, s);
}

// One layer of forward_network_gpu's loop (src/network.c:772-785), over part of the batch.
static int forward_layer(dnb_network *net, int i, const float *device_input, const Part &p, cudaStream_t s)
{
    Layer &L = net->layers[i];
    dnb_tensor in;
    if (i == 0) {
        in = dnb_tensor{(void *)device_input, DNB_NCHW, DNB_F32, net->batch, net->c, net->h, net->w, 0};
        if (net->input_nhwc.data) in = net->input_nhwc;   // filled by prepare_input
    } else {
        in = net->layers[i - 1].out;
    }
    in = part_of(in, p);
    const dnb_tensor out = part_of(L.out, p);
    switch (L.kind) {
    case L_CONV:
        if (L.fuses_next_shortcut) {
            Layer &S = net->layers[i + 1];
            const dnb_tensor add = part_of(net->layers[S.from].out, p), sum = part_of(S.out, p);
            return conv_shortcut_general(plan_of(L, p), &in, &add, &sum, S.alpha, S.beta, S.activation, s);
        }
        if (L.fuses_next_pool) {
            // The first layer's own output is made from the images, if it is asked for: those of a caller may be gone by then, so they are copied.
            // conv_stem_rows.cu does it on the way (Darknet-19-xnor, 128 images: 1057 us a step, 1073 with a copy before it), the other kernel for
            // few images, for which a copy is mostly a launch (YOLOv3-tiny, one: 131 and 134; 16: 439 and 432).
            float *keep = nullptr;
            if (i == 0 && device_input != net->input_slot[0] && device_input != net->input_slot[1]) {
                const size_t bytes = (size_t)net->batch * net->inputs * sizeof(float);
                // (an xnor layer that comes first has no kernel that writes the copy)
                if (L.plan->stem_tc && (L.plan->keep_k_order || bytes <= (size_t)8 << 20)) keep = net->input_dev;
                else DNB_CUDA(cudaMemcpyAsync(net->input_dev, device_input, bytes, cudaMemcpyDeviceToDevice, s));
            }
            const dnb_tensor pooled = part_of(net->layers[i + 1].out, p);
            return conv_pool_forward(plan_of(L, p), &in, &pooled, keep, s);
        }
        if (L.fuses_next_yolo) {
            Layer &Y = net->layers[i + 1];
            const dnb_tensor head = part_of(Y.out, p);
            return dnb_conv_yolo_forward(plan_of(L, p), &in, &head, Y.anchors, Y.classes, s);
        }
        return dnb_conv_forward(plan_of(L, p), &in, &out, nullptr, s);
    case L_CONNECTED: {
        // forward_connected_layer_gpu (src/connected_layer.c:288-306): the previous layer's whole channels-last output
        // is one pixel of h*w*cpitch channels per image
        dnb_tensor flat = in;
        flat.h = flat.w = 1;
        flat.c = flat.cpitch = L.cd.c;
        return dnb_conv_forward(plan_of(L, p), &flat, &out, nullptr, s);
    }
    case L_MAXPOOL:
        if (L.fused_into_prev) return DNB_OK;   // done by the convolution before it
        return launch_maxpool(&in, &out, L.size, L.stride, L.padding, s, L.sign_out, L.sign_pitch);
    case L_UPSAMPLE: return launch_upsample(&in, &out, L.stride, L.scale, s);
    case L_SHORTCUT: {
        if (L.fused_into_prev) return DNB_OK;   // done by the convolution before it
        const dnb_tensor add = part_of(net->layers[L.from].out, p);
        return launch_shortcut(&in, &add, &out, L.alpha, L.beta, L.activation, s);
    }
    case L_ROUTE: {
        std::vector<dnb_tensor> parts;
        for (int id : L.inputs) parts.push_back(part_of(net->layers[id].out, p));
        std::vector<const dnb_tensor *> ins;
        for (const dnb_tensor &t : parts) ins.push_back(&t);
        return launch_route(ins.data(), (int)ins.size(), &out, s);
    }
    case L_YOLO:
        if (L.fused_into_prev) return DNB_OK;   // done by the convolution before it
        return launch_convert(&in, &out, 0, L.anchors, L.classes, s);
    case L_AVGPOOL: return launch_avgpool(&in, &out, s);
    case L_SOFTMAX: return launch_softmax(&in, &out, L.groups, L.temperature, s);
    }
    return DNB_OK;
}

static int forward_eager(dnb_network *net, const float *device_input, cudaStream_t s)
{
    const Part all = whole(net);
    DNB_TRY(prepare_input(net, device_input, all, s));
    for (int i = 0; i < (int)net->layers.size(); ++i) DNB_TRY(forward_layer(net, i, device_input, all, s));
    return DNB_OK;
}

// The captured device-resident forward, which belongs to one input and stream.
static void drop_forward_graph(dnb_network *net)
{
    if (net->graph_exec) cudaGraphExecDestroy(net->graph_exec);
    net->graph_exec = nullptr;
    net->graph_input = nullptr;
    net->graph_stream = nullptr;
    net->eager_runs = 0;
}

// ... and everything else that holds the parameters' pointers or the plans' launch blocks: the captured steps, which read the
// network's own input buffers whatever forward is given, and the plans of parts of a batch.
static void drop_graph(dnb_network *net)
{
    drop_forward_graph(net);
    for (int k = 0; k < 2; ++k) {
        if (net->step_exec[k]) cudaGraphExecDestroy(net->step_exec[k]);
        net->step_exec[k] = nullptr;
        net->step_runs[k] = 0;
        for (cudaGraphExec_t e : net->item_exec[k]) if (e) cudaGraphExecDestroy(e);
        net->item_exec[k].clear();
    }
    for (Layer &L : net->layers)
        for (dnb_conv_plan *&q : L.piece_plan) { dnb_conv_plan_destroy(q); q = nullptr; }
}

extern "C" int dnb_network_enable_graph(dnb_network *net, int on)
{
    if (!net) DNB_FAIL(DNB_EINVAL, "enable_graph: null network");
    net->graph_enabled = on != 0;
    if (!on) drop_forward_graph(net);
    return DNB_OK;
}

extern "C" int dnb_network_forward(dnb_network *net, const float *device_input, void *stream)
{
    if (!net || !device_input) DNB_FAIL(DNB_EINVAL, "network_forward: null argument");
    if (!net->weights_loaded) DNB_FAIL(DNB_EINVAL, "network_forward: load_weights has not been called");
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "network_forward: a submitted step is still in flight (the layers' outputs are shared); collect it first");
    DNB_TRY(check_current_device(net->device, "network_forward"));
    point_status(net, 0);
    net->images = net->input_dev;
    cudaStream_t s = (cudaStream_t)stream;  // NULL is the legacy default stream, as everywhere in CUDA
    if (!net->graph_enabled || !s) return forward_eager(net, device_input, s);   // the legacy stream cannot be captured

    // Graph replay: at small batches the 100-odd launches of a forward pass cost more than its kernels.  The
    // first forward with a given (input, stream) runs eagerly (plans build their tensor maps and scratch then),
    // the second is captured, every later one is a single cudaGraphLaunch.
    if (net->graph_exec && net->graph_input == device_input && net->graph_stream == s) {
        DNB_CUDA(cudaGraphLaunch(net->graph_exec, s));
        return DNB_OK;
    }
    if (net->graph_input != device_input || net->graph_stream != s) {
        drop_forward_graph(net);
        net->graph_input = device_input;
        net->graph_stream = s;
    }
    if (net->eager_runs++ == 0) return forward_eager(net, device_input, s);
    cudaGraph_t graph = nullptr;
    DNB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int rc = forward_eager(net, device_input, s);
    const cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (rc != DNB_OK || ce != cudaSuccess || !graph) {
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        net->graph_enabled = false;          // something on the path cannot be captured: stay eager from here on
        drop_forward_graph(net);
        return forward_eager(net, device_input, s);
    }
    const cudaError_t ie = cudaGraphInstantiate(&net->graph_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
        cudaGetLastError();
        net->graph_exec = nullptr;
        net->graph_enabled = false;
        return forward_eager(net, device_input, s);
    }
    DNB_CUDA(cudaGraphLaunch(net->graph_exec, s));
    return DNB_OK;
}

extern "C" int dnb_conv_plan_check_status(dnb_conv_plan *p);

// The second set of buffers exists only once two steps are in flight.
static int ensure_second_slot(dnb_network *net)
{
    if (net->input_slot[1]) return DNB_OK;
    DNB_CUDA(cudaMalloc((void **)&net->input_slot[1], (size_t)net->batch * net->inputs * sizeof(float)));
    DNB_CUDA(cudaMallocHost((void **)&net->out_host_slot[1], (size_t)net->batch * net->outputs * sizeof(float)));
    for (Layer &L : net->layers)
        if (L.kind == L_YOLO && !L.host_slot[1]) DNB_CUDA(cudaMallocHost((void **)&L.host_slot[1], tensor_elems(&L.out) * sizeof(float)));
    return DNB_OK;
}

// The batch's images to the device.  Page-locked memory goes straight to the copy engine; ordinary memory, where Darknet's
// own loaders keep images, is carried over by a few threads (host_copy.cu) and has been read when this returns.  A network's first
// steps make no ring of page-locked memory of their own, but use the process's if there is one: it takes as long as a first step
// (ResNet-50, one image, alone: first call 14.2 ms with a ring made in it, 1.0 without), and only a program that goes on gains by it.
static int upload(dnb_network *net, const float *input, float *in_dev, int images, cudaStream_t s)
{
    const size_t bytes = (size_t)images * net->inputs * sizeof(float);
    cudaPointerAttributes at;
    const bool known = cudaPointerGetAttributes(&at, input) == cudaSuccess;
    if (!known) cudaGetLastError();
    if (known && at.type != cudaMemoryTypeUnregistered) {
        DNB_CUDA(cudaMemcpyAsync(in_dev, input, bytes, cudaMemcpyHostToDevice, s));
        return DNB_OK;
    }
    if (!net->copier) net->copier = copy_pool(net->submitted >= STAGED_FROM);
    const int rc = upload_staged(net->copier.get(), in_dev, input, bytes, (size_t)net->batch * net->inputs * sizeof(float), s);
    if (rc != NOT_STAGED) return rc;
    DNB_CUDA(cudaMemcpyAsync(in_dev, input, bytes, cudaMemcpyHostToDevice, s));
    return DNB_OK;
}

// The layers up to and including the next [yolo] layer, or the last layer, from layer `begin` on.
static int segment_end(const dnb_network *net, int begin)
{
    int i = begin;
    while (i + 1 < (int)net->layers.size() && net->layers[i].kind != L_YOLO) ++i;
    return i + 1;
}

static int enqueue_segment(dnb_network *net, int slot, int begin, int end, const Part &p, cudaStream_t s)
{
    float *in_dev = net->input_slot[slot];
    if (begin == 0) DNB_TRY(prepare_input(net, in_dev, p, s));
    for (int i = begin; i < end; ++i) DNB_TRY(forward_layer(net, i, in_dev, p, s));
    Layer &last = net->layers.back();
    if (end == (int)net->layers.size() && last.kind != L_YOLO) {
        const dnb_tensor y = part_of(last.out, p), o = part_of(dnb_tensor{net->out_dev_nchw, DNB_NCHW, DNB_F32, net->batch, last.out_c, last.out_h, last.out_w, 0}, p);
        DNB_TRY(launch_convert(&y, &o, 0, 0, 0, s));
    }
    return DNB_OK;
}

// Captures what `enqueue` puts on s into *exec and launches it.  False, with nothing enqueued: something on the path cannot
// be captured, eager from here on.
template <typename F>
static bool launch_captured(dnb_network *net, cudaGraphExec_t *exec, cudaStream_t s, F enqueue)
{
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) { cudaGetLastError(); return false; }
    const int rc = enqueue();
    const cudaError_t ce = cudaStreamEndCapture(s, &graph);
    cudaError_t ie = cudaErrorUnknown;
    if (rc == DNB_OK && ce == cudaSuccess && graph) ie = cudaGraphInstantiate(exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (ie == cudaSuccess && cudaGraphLaunch(*exec, s) == cudaSuccess) return true;
    cudaGetLastError();
    if (ie == cudaSuccess) cudaGraphExecDestroy(*exec);
    *exec = nullptr;
    net->step_graphs = false;
    return false;
}

// One item of a step: its layers (forward_network_gpu's loop, src/network.c:772-785) on the compute stream, and, where it ends
// in a [yolo] layer or the output layer, that layer's pull (src/yolo_layer.c:360, src/network.c:786) on the copy stream while
// the following layers compute.  Every device-to-host copy goes through the copy stream: a copy enqueued on the compute stream
// would queue behind the large [yolo] pulls on the copy engine and hold back the next step's layers.
// alone: no other step is in flight, so there is nobody to wait for and nobody who waits.
// exec: where the item's graph is kept, null for plain launches.
static int enqueue_item(dnb_network *net, int slot, const Item &it, bool alone, cudaGraphExec_t *exec)
{
    cudaStream_t s = net->stream, cs = net->copy_stream;
    const bool wait = !alone && net->submitted > 0;
    const Part &p = it.part;
    const int k = p.piece < 0 ? 0 : p.piece;
    Layer &L = net->layers[it.end - 1];
    const bool output = it.end == (int)net->layers.size() && L.kind != L_YOLO;
    // the previous step's pull has read what this item's last layer, or the convolution that does its work, overwrites
    if (wait && L.kind == L_YOLO) DNB_CUDA(cudaStreamWaitEvent(s, L.copied[k], 0));
    if (wait && output) DNB_CUDA(cudaStreamWaitEvent(s, net->copy_done[slot ^ 1], 0));
    if (exec && *exec) DNB_CUDA(cudaGraphLaunch(*exec, s));
    else if (!exec || !net->step_graphs || !launch_captured(net, exec, s, [&]() { return enqueue_segment(net, slot, it.begin, it.end, p, s); }))
        DNB_TRY(enqueue_segment(net, slot, it.begin, it.end, p, s));
    if (L.kind != L_YOLO && !output) return DNB_OK;
    cudaEvent_t ready = output ? net->fwd_done[slot] : L.done;
    DNB_CUDA(cudaEventRecord(ready, s));
    DNB_CUDA(cudaStreamWaitEvent(cs, ready, 0));
    if (output) {
        const size_t first = (size_t)p.first * net->outputs;
        DNB_CUDA(cudaMemcpyAsync(net->out_host_slot[slot] + first, net->out_dev_nchw + first, (size_t)p.count * net->outputs * sizeof(float), cudaMemcpyDeviceToHost, cs));
        return DNB_OK;
    }
    const dnb_tensor out = part_of(L.out, p);
    DNB_CUDA(cudaMemcpyAsync(L.host_slot[slot] + tensor_elems(&L.out) / net->batch * p.first, out.data, tensor_elems(&out) * sizeof(float), cudaMemcpyDeviceToHost, cs));
    if (!alone) DNB_CUDA(cudaEventRecord(L.copied[k], cs));
    return DNB_OK;
}

// After the last item.  alone: the streams are joined.
static int finish_step(dnb_network *net, int slot, bool alone)
{
    cudaStream_t s = net->stream, cs = net->copy_stream;
    DNB_CUDA(cudaMemcpyAsync(net->status_host + slot, net->status_dev + slot, sizeof(int), cudaMemcpyDeviceToHost, cs));
    if (alone) {
        DNB_CUDA(cudaEventRecord(net->pulled, cs));
        DNB_CUDA(cudaStreamWaitEvent(s, net->pulled, 0));
    }
    return DNB_OK;
}

// A step whose images are on the device, or will be where the compute stream stands.
static int enqueue_step(dnb_network *net, int slot, bool alone)
{
    point_status(net, slot);
    for (int begin = 0, end; begin < (int)net->layers.size(); begin = end) {
        end = segment_end(net, begin);
        DNB_TRY(enqueue_item(net, slot, Item{begin, end, whole(net), false}, alone, nullptr));
    }
    return finish_step(net, slot, alone);
}

// A step by its schedule, uploads included.  The first step of a slot runs eagerly, the second is captured item by item.
static int enqueue_schedule(dnb_network *net, int slot, const float *input, bool alone)
{
    const bool graphs = net->step_graphs && net->step_runs[slot]++ > 0;
    if (graphs) net->item_exec[slot].resize(net->schedule.size(), nullptr);
    point_status(net, slot);
    for (size_t i = 0; i < net->schedule.size(); ++i) {
        const Item &it = net->schedule[i];
        if (it.uploads) {
            const size_t first = (size_t)it.part.first * net->inputs;
            cudaEvent_t in = net->piece_in[it.part.piece < 0 ? 0 : it.part.piece];
            DNB_TRY(upload(net, input + first, net->input_slot[slot] + first, it.part.count, net->h2d_stream));
            DNB_CUDA(cudaEventRecord(in, net->h2d_stream));
            DNB_CUDA(cudaStreamWaitEvent(net->stream, in, 0));
        }
        DNB_TRY(enqueue_item(net, slot, it, alone, graphs ? &net->item_exec[slot][i] : nullptr));
    }
    return finish_step(net, slot, alone);
}

// Whether, and how, a step's batch is cut into parts.  With a copy engine at about 50 GB/s the images of a large batch are on
// their way for as long as a good part of the layers takes, and so are the results of the last [yolo] layer, the largest
// map; with the whole batch as one unit neither overlaps anything within a step.
//  * front: the first layers run part by part, each as soon as its images are there.  Only layers that fill the chip with a part
//    of the batch (two waves of 128 x 128 tiles), as many as the upload takes time.
//  * tail: the last layers run in two halves, so that the first half's results are pulled while the second computes.  Deep
//    layers lose by it, about 6 us each (half a wave, a launch), measured: YOLOv3-608 in TF32 takes 18.16 ms at batch 64,
//    2 x 9.30 at 32, 2 x 4.92 of 9.30 at 16; so the tail is as long as pays.
// The layers' times are estimates from their operations and bytes at the rates the kernels reach.  Networks with xnor
// layers, whose kernels hand each other whole-batch sign tensors, run uncut.
// Measured: YOLOv3-416, 8 images, bf16, one blocking step 2358 -> 2113 us; YOLOv3-608 in TF32, two steps of 64 images in flight
// 46.0 -> 43.1 ms.
static void plan_step(dnb_network *net)
{
    const double copy_rate = 50e3, byte_rate = 4e6;   // bytes per us
    const double tc_rate = net->mode == DNB_MODE_BF16 ? 1.0e9 : net->mode == DNB_MODE_TF32 ? 5.4e8 : 1.1e8, cuda_core_rate = 3e7;   // operations per us
    const double part_us = 4, half_us = 6, worth_us = 50;
    const int n = (int)net->layers.size(), batch = net->batch;
    net->schedule.clear();
    std::vector<double> us(n);
    for (int i = 0; i < n; ++i) {
        const Layer &L = net->layers[i];
        if (L.kind == L_CONV && L.cd.xnor) return;
        double ops = 0;
        if (L.kind == L_CONV) ops = 2.0 * L.cd.n * L.cd.size * L.cd.size * (L.cd.c / L.cd.groups) * L.out_h * L.out_w * batch;
        const double written = (double)L.out_c * L.out_h * L.out_w / (L.fuses_next_pool ? 4 : 1);
        const double bytes = L.fused_into_prev ? 0 : ((double)L.c * L.h * L.w + written) * batch * elem_size(net->dtype);
        const bool cuda_cores = net->mode == DNB_MODE_FP32 && L.plan && !L.plan->fp32_tc;
        us[i] = std::max(ops / (cuda_cores ? cuda_core_rate : tc_rate), bytes / byte_rate);
    }
    // every tensor that layer i reads or writes has its part where the kernels' alignment rules want it
    auto aligned = [&](const dnb_tensor &t, int each) {
        return !t.data || tensor_elems(&t) / t.n * each * elem_size(t.dtype) % (t.layout == DNB_NHWC ? 128 : 16) == 0;
    };
    auto divisible = [&](int i, int each) {
        const Layer &L = net->layers[i];
        bool ok = aligned(L.out, each) && (i > 0 ? aligned(net->layers[i - 1].out, each) : aligned(net->input_nhwc, each) && (size_t)each * net->inputs % 4 == 0);
        if (L.kind == L_SHORTCUT) ok = ok && aligned(net->layers[L.from].out, each);
        for (int id : L.inputs) ok = ok && aligned(net->layers[id].out, each);
        return ok;
    };
    auto cuttable = [&](int i) { return i > 0 && i < n && !net->layers[i - 1].fuses_next_shortcut && !net->layers[i - 1].fuses_next_yolo && !net->layers[i - 1].fuses_next_pool; };

    const double upload_us = (double)batch * net->inputs * sizeof(float) / copy_rate;
    int front = 0, parts = 1;
    double best = worth_us;
    for (int k = 2; k <= MAX_PIECES && batch % k == 0; k *= 2) {
        const int each = batch / k;
        double t = 0;
        for (int i = 0; i < n && t < upload_us; ++i) {
            const Layer &L = net->layers[i];
            const double blocks = std::ceil((double)each * L.out_h * L.out_w / 128) * ((L.out_c + 127) / 128);
            if (L.kind == L_YOLO || L.kind == L_CONNECTED || blocks < 2.0 * sm_count() || !divisible(i, each)) break;
            t += us[i];
            const double saved = std::min(t, upload_us) * (1 - 1.0 / k) - part_us * (i + 1) * (k - 1);
            if (cuttable(i + 1) && saved > best) { best = saved; front = i + 1; parts = k; }
        }
    }

    int tail = n;
    if (net->layers[n - 1].kind == L_YOLO && batch % 2 == 0) {
        const double pull_us = (double)tensor_elems(&net->layers[n - 1].out) * sizeof(float) / copy_rate;
        double t = 0;
        best = worth_us;
        for (int i = n - 1; i > front && divisible(i, batch / 2); --i) {
            t += us[i];
            const double saved = std::min(t, pull_us) / 2 - half_us * (n - i);
            if (cuttable(i) && saved > best) { best = saved; tail = i; }
        }
    }
    if (!front && tail == n) return;

    for (int k = 0; k < parts && front; ++k) net->schedule.push_back(Item{0, front, Part{k * (batch / parts), batch / parts, k}, true});
    for (int begin = front, end; begin < tail; begin = end) {
        end = std::min(segment_end(net, begin), tail);
        net->schedule.push_back(Item{begin, end, whole(net), begin == 0});
    }
    for (int h = 0; h < 2 && tail < n; ++h)
        for (int begin = tail, end; begin < n; begin = end) {
            end = segment_end(net, begin);
            net->schedule.push_back(Item{begin, end, Part{h * (batch / 2), batch / 2, h}, false});
        }
}
static int check_step(dnb_network *net, const float *input, const char *what)
{
    if (!net || !input) DNB_FAIL(DNB_EINVAL, "%s: null argument", what);
    if (!net->weights_loaded) DNB_FAIL(DNB_EINVAL, "%s: load_weights has not been called", what);
    return check_current_device(net->device, what);
}

// Enqueues one step.  Up to two steps may be in flight, so the copies of one step overlap the layers of the next.
extern "C" int dnb_network_submit(dnb_network *net, const float *input)
{
    if (net && net->submitted - net->collected >= 2) DNB_FAIL(DNB_EINVAL, "network_submit: two steps are already in flight; collect one first");
    DNB_TRY(check_step(net, input, "network_submit"));
    const int slot = (int)(net->submitted & 1);
    if (slot == 1) DNB_TRY(ensure_second_slot(net));
    // the slot's buffers are free: the step that used them last has been collected
    if (!net->schedule.empty()) {
        DNB_TRY(enqueue_schedule(net, slot, input, false));
    } else {
        DNB_TRY(upload(net, input, net->input_slot[slot], net->batch, net->h2d_stream));
        DNB_CUDA(cudaEventRecord(net->in_ready[slot], net->h2d_stream));
        DNB_CUDA(cudaStreamWaitEvent(net->stream, net->in_ready[slot], 0));
        DNB_TRY(enqueue_step(net, slot, false));
    }
    DNB_CUDA(cudaEventRecord(net->copy_done[slot], net->copy_stream));
    ++net->submitted;
    return DNB_OK;
}

// Waits for the oldest step in flight and hands out its results.
extern "C" int dnb_network_collect(dnb_network *net, float **output)
{
    if (!net || !output) DNB_FAIL(DNB_EINVAL, "network_collect: null argument");
    if (net->submitted == net->collected) DNB_FAIL(DNB_EINVAL, "network_collect: nothing has been submitted");
    const int slot = (int)(net->collected & 1);
    ++net->collected;
    net->images = net->input_slot[slot];
    DNB_CUDA(cudaEventSynchronize(net->copy_done[slot]));   // follows fwd_done[slot] and every copy of the step
    for (Layer &L : net->layers) if (L.kind == L_YOLO) L.host_out = L.host_slot[slot];
    if (net->status_host[slot]) {
        // this step's own word: the other step in flight keeps its word and its verdict
        const int code = net->status_host[slot];
        net->status_host[slot] = 0;
        cudaMemsetAsync(net->status_dev + slot, 0, sizeof(int), net->stream);   // before the slot's next step, which follows on this stream
        char text[512];
        snprintf(text, sizeof(text), kTimeoutText, code);
        DNB_FAIL(DNB_ETIMEOUT, "network_predict: %s", text);
    }
    Layer &last = net->layers.back();
    *output = last.kind == L_YOLO ? last.host_out : net->out_host_slot[slot];
    return DNB_OK;
}

// network_predict (src/network.c:497-508): one step, start to finish.  At small batches the hundred-odd launches of a step
// cost the host more than the device needs for it, and nothing overlaps them in a blocking call.  So the first step of a
// slot runs eagerly (plans build their tensor maps and scratch then), the second is captured, copies included, and every
// later one is the upload and one graph launch.  (YOLOv3-tiny-416, one image: the host spent 100 us on a step's launches.)
extern "C" int dnb_network_predict(dnb_network *net, const float *input, float **output)
{
    if (!net || !input || !output) DNB_FAIL(DNB_EINVAL, "network_predict: null argument");
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "network_predict: a submitted step has not been collected");
    DNB_TRY(check_step(net, input, "network_predict"));
    const int slot = (int)(net->submitted & 1);
    if (slot == 1) DNB_TRY(ensure_second_slot(net));
    cudaStream_t s = net->stream;
    if (!net->schedule.empty()) {
        DNB_TRY(enqueue_schedule(net, slot, input, true));
    } else {
        DNB_TRY(upload(net, input, net->input_slot[slot], net->batch, s));
        if (net->step_exec[slot]) DNB_CUDA(cudaGraphLaunch(net->step_exec[slot], s));
        else if (!net->step_graphs || net->step_runs[slot]++ == 0 || !launch_captured(net, &net->step_exec[slot], s, [&]() { return enqueue_step(net, slot, true); }))
            DNB_TRY(enqueue_step(net, slot, true));
    }
    DNB_CUDA(cudaEventRecord(net->copy_done[slot], s));
    ++net->submitted;
    return dnb_network_collect(net, output);
}

extern "C" int dnb_network_num_layers(const dnb_network *net) { return net ? (int)net->layers.size() : 0; }
extern "C" int dnb_network_batch(const dnb_network *net) { return net ? net->batch : 0; }
extern "C" int dnb_network_inputs(const dnb_network *net) { return net ? net->inputs : 0; }
extern "C" int dnb_network_outputs(const dnb_network *net) { return net ? net->outputs : 0; }

extern "C" int dnb_network_layer_shape(const dnb_network *net, int i, int *c, int *h, int *w)
{
    if (!net || i < 0 || i >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "layer index %d out of range", i);
    if (c) *c = net->layers[i].out_c;
    if (h) *h = net->layers[i].out_h;
    if (w) *w = net->layers[i].out_w;
    return DNB_OK;
}
extern "C" const char *dnb_network_layer_type(const dnb_network *net, int i)
{
    return (!net || i < 0 || i >= (int)net->layers.size()) ? "" : kKindNames[net->layers[i].kind];
}
extern "C" const char *dnb_network_layer_kernel(const dnb_network *net, int i)
{
    if (!net || i < 0 || i >= (int)net->layers.size()) return "";
    const Layer &L = net->layers[i];
    return L.plan ? dnb_conv_plan_kernel(L.plan) : kKindNames[L.kind];
}

// Images [first, first + count) of layer i's output, NCHW f32, to the host.
extern "C" int dnb_conv_plan_describe(const dnb_conv_plan *p, char *buf, int len);

extern "C" int dnb_network_layer_describe(const dnb_network *net, int i, char *buf, int len)
{
    if (!net || !buf || len < 1 || i < 0 || i >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "layer_describe: bad argument");
    const Layer &L = net->layers[i];
    if (L.plan) return dnb_conv_plan_describe(L.piece_plan[0] && !L.plan->tc_x_ptr ? L.piece_plan[0] : L.plan, buf, len);   // a layer that only ran in parts
    snprintf(buf, len, "%s%s", kKindNames[L.kind], L.fused_into_prev ? " fused" : "");
    return DNB_OK;
}

extern "C" int dnb_network_layer_output_images(dnb_network *net, int i, int first, int count, float *host_out)
{
    if (!net || !host_out || i < 0 || i >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "layer_output: bad argument");
    if (first < 0 || count < 1 || first + count > net->batch) DNB_FAIL(DNB_EINVAL, "layer_output: images %d..%d of a batch of %d", first, first + count - 1, net->batch);
    Layer &L = net->layers[i];
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "layer_output: a submitted step is still in flight; collect it first");
    if (!L.out.data && !L.own_out.data)
        DNB_FAIL(DNB_EUNSUPPORTED, "layer %d is fused into layer %d and has no output of its own (DNB_FUSE_SHORTCUT=0 / DNB_FUSE_YOLO=0 keep it)", i, i + 1);
    const size_t per_image = (size_t)L.out_c * L.out_h * L.out_w;
    const size_t elems = (size_t)count * per_image;
    DNB_CUDA(cudaDeviceSynchronize());  // the forward may have run on any stream
    if (L.out.layout == DNB_NCHW) {
        DNB_CUDA(cudaMemcpy(host_out, (const float *)L.out.data + (size_t)first * per_image, elems * sizeof(float), cudaMemcpyDeviceToHost));
        return DNB_OK;
    }
    // a run of whole images of a channels-last tensor is itself a channels-last tensor, if it starts on a 128-byte
    // boundary; where it does not (small maps with odd pitches) the whole layer is converted and the run copied out
    const size_t image_bytes = (size_t)L.out_h * L.out_w * L.out.cpitch * elem_size(L.out.dtype);
    const bool aligned = ((size_t)first * image_bytes) % 128 == 0;
    const int conv_first = aligned ? first : 0, conv_count = aligned ? count : net->batch;
    const size_t conv_elems = (size_t)conv_count * per_image;
    if (conv_elems > net->export_elems) {
        cudaFree(net->export_dev);
        net->export_dev = nullptr; net->export_elems = 0;
        DNB_CUDA(cudaMalloc((void **)&net->export_dev, conv_elems * sizeof(float)));
        net->export_elems = conv_elems;
    }
    dnb_tensor in;
    DNB_TRY(own_output(net, i, &in, net->stream));
    in.n = conv_count;
    in.data = (char *)in.data + (size_t)conv_first * image_bytes;
    dnb_tensor o{net->export_dev, DNB_NCHW, DNB_F32, conv_count, L.out_c, L.out_h, L.out_w, 0};
    DNB_TRY(launch_convert(&in, &o, 0, 0, 0, net->stream));
    DNB_CUDA(cudaStreamSynchronize(net->stream));
    DNB_CUDA(cudaMemcpy(host_out, net->export_dev + (size_t)(first - conv_first) * per_image, elems * sizeof(float), cudaMemcpyDeviceToHost));
    return DNB_OK;
}

extern "C" int dnb_network_layer_output(dnb_network *net, int i, float *host_out)
{
    if (!net) DNB_FAIL(DNB_EINVAL, "layer_output: bad argument");
    return dnb_network_layer_output_images(net, i, 0, net->batch, host_out);
}

// Waits for the device, then reads and clears both status words: DNB_ETIMEOUT if a bounded wait expired in any
// convolution since the last check.  For callers of the device-resident dnb_network_forward, which returns
// before its kernels have run; dnb_network_collect reports the same for submitted steps.
extern "C" int dnb_network_check_status(dnb_network *net)
{
    if (!net) DNB_FAIL(DNB_EINVAL, "check_status: null network");
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "check_status: a submitted step is still in flight; collect it first");
    int v[2] = {0, 0};
    DNB_CUDA(cudaDeviceSynchronize());
    DNB_CUDA(cudaMemcpy(v, net->status_dev, sizeof(v), cudaMemcpyDeviceToHost));
    if (v[0] || v[1]) {
        DNB_CUDA(cudaMemset(net->status_dev, 0, sizeof(v)));
        char text[512];
        snprintf(text, sizeof(text), kTimeoutText, v[0] ? v[0] : v[1]);
        DNB_FAIL(DNB_ETIMEOUT, "network_forward: %s", text);
    }
    return DNB_OK;
}

extern "C" int dnb_conv_plan_set_diagnostics(dnb_conv_plan *p, long long wait_limit_cycles, int debug_bits);

// dnb_conv_plan_set_diagnostics for convolution `layer` of the network.
extern "C" int dnb_network_set_diagnostics(dnb_network *net, int layer, long long wait_limit_cycles, int debug_bits)
{
    if (!net || layer < 0 || layer >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "set_diagnostics: bad argument");
    Layer &L = net->layers[layer];
    if (L.kind != L_CONV) DNB_FAIL(DNB_EINVAL, "set_diagnostics: layer %d is not convolutional", layer);
    // launches already enqueued carry their own copy of the argument block: only later ones see the change
    drop_graph(net);
    return dnb_conv_plan_set_diagnostics(L.plan, wait_limit_cycles, debug_bits);
}

extern "C" int dnb_network_yolo_output(dnb_network *net, int i, const float **host_out)
{
    if (!net || !host_out || i < 0 || i >= (int)net->layers.size()) DNB_FAIL(DNB_EINVAL, "yolo_output: bad argument");
    if (net->layers[i].kind != L_YOLO) DNB_FAIL(DNB_EINVAL, "layer %d is not a [yolo] layer", i);
    *host_out = net->layers[i].host_out;
    return DNB_OK;
}

// numops (examples/darknet.c:81-114): 2 * n * size^2 * c/groups * out_h * out_w per convolution and image.
extern "C" double dnb_network_flops(const dnb_network *net)
{
    double ops = 0;
    if (!net) return 0;
    for (const Layer &L : net->layers)
        if (L.kind == L_CONV)
            ops += 2.0 * L.cd.n * L.cd.size * L.cd.size * (L.cd.c / L.cd.groups) * L.out_h * L.out_w;
        else if (L.kind == L_CONNECTED)
            ops += 2.0 * L.fc_inputs * L.cd.n;   // examples/darknet.c:91-92
    return ops * net->batch;
}

extern "C" int dnb_network_launches(const dnb_network *net)
{
    int n = 0;
    if (!net) return 0;
    for (const Layer &L : net->layers) n += L.launches;
    if (net->input_nhwc.data) n += 1;
    return n;
}

// Forward with a CUDA event between layers, asynchronous like dnb_network_forward.  `slot` selects an
// independent set of events so that several timed forwards can be in flight before any is read.
extern "C" int dnb_network_forward_timed(dnb_network *net, const float *device_input, void *stream, int slot)
{
    if (!net || !device_input || slot < 0 || slot > 4096) DNB_FAIL(DNB_EINVAL, "network_forward_timed: bad argument");
    if (!net->weights_loaded) DNB_FAIL(DNB_EINVAL, "network_forward_timed: load_weights has not been called");
    if (net->submitted != net->collected) DNB_FAIL(DNB_EINVAL, "network_forward_timed: a submitted step is still in flight; collect it first");
    DNB_TRY(check_current_device(net->device, "network_forward_timed"));
    point_status(net, 0);
    net->images = net->input_dev;
    const int n = (int)net->layers.size();
    while ((int)net->events.size() < (slot + 1) * (n + 1)) {
        cudaEvent_t e;
        DNB_CUDA(cudaEventCreate(&e));
        net->events.push_back(e);
    }
    cudaStream_t s = (cudaStream_t)stream;
    cudaEvent_t *ev = &net->events[(size_t)slot * (n + 1)];
    DNB_TRY(prepare_input(net, device_input, whole(net), s));   // outside the per-layer brackets: layer 0's time is its kernel's
    for (int i = 0; i < n; ++i) {
        DNB_CUDA(cudaEventRecord(ev[i], s));
        DNB_TRY(forward_layer(net, i, device_input, whole(net), s));
    }
    DNB_CUDA(cudaEventRecord(ev[n], s));
    return DNB_OK;
}

// Per-layer device time of the timed forward in `slot`, milliseconds; waits for that forward to finish.
extern "C" int dnb_network_timed_ms(dnb_network *net, int slot, float *layer_ms)
{
    if (!net || !layer_ms || slot < 0) DNB_FAIL(DNB_EINVAL, "network_timed_ms: bad argument");
    const int n = (int)net->layers.size();
    if ((int)net->events.size() < (slot + 1) * (n + 1)) DNB_FAIL(DNB_EINVAL, "network_timed_ms: slot %d was never recorded", slot);
    cudaEvent_t *ev = &net->events[(size_t)slot * (n + 1)];
    DNB_CUDA(cudaEventSynchronize(ev[n]));
    for (int i = 0; i < n; ++i) DNB_CUDA(cudaEventElapsedTime(&layer_ms[i], ev[i], ev[i + 1]));
    return DNB_OK;
}

extern "C" int dnb_network_profile(dnb_network *net, const float *device_input, float *layer_ms)
{
    DNB_TRY(dnb_network_forward_timed(net, device_input, net->stream, 0));
    return dnb_network_timed_ms(net, 0, layer_ms);
}
