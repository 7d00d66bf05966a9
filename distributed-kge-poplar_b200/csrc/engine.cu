// Host engine implementation.  See engine.hpp.
#include "engine.hpp"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <optional>
#include <utility>

namespace kge {

// ---------------------------------------------------------------------------
// Settings (src/poplar_kge.cpp:39-67 for the error texts, :198-246 for the keys)

namespace {

const char* type_name(int type) {
    switch (type) {
        case KGE_SET_STRING: return "string";
        case KGE_SET_BOOL: return "bool";
        case KGE_SET_FLOAT: return "float";
        case KGE_SET_UNSIGNED: return "unsigned";
    }
    return "?";
}

const SettingValue& lookup(const SettingMap& s, const std::string& key, int type) {
    auto it = s.find(key);
    if (it == s.end()) fail(KGE_INVALID_ARGUMENT, msg() << "Key not found '" << key << "'");
    if (it->second.type != type) {
        fail(KGE_INVALID_ARGUMENT, msg() << "Key '" << key
                                         << "' holds value of unexpected type. Expected: '"
                                         << type_name(type) << "', actual: '"
                                         << type_name(it->second.type) << "'.");
    }
    return it->second;
}
std::string get_string(const SettingMap& s, const std::string& k) { return lookup(s, k, KGE_SET_STRING).s; }
unsigned get_unsigned(const SettingMap& s, const std::string& k) {
    return (unsigned)lookup(s, k, KGE_SET_UNSIGNED).u;
}
float get_float(const SettingMap& s, const std::string& k) { return (float)lookup(s, k, KGE_SET_FLOAT).f; }
bool get_bool(const SettingMap& s, const std::string& k) { return lookup(s, k, KGE_SET_BOOL).u != 0; }

template <class T, class Getter>
T get_or(const SettingMap& s, const std::string& k, Getter getter, T fallback) {
    return s.count(k) ? getter(s, k) : fallback;
}

int parse_storage(const std::string& key, const std::string& value) {
    if (value == "float32") return ST_F32;
    if (value == "float16") return ST_F16;
    fail(KGE_INVALID_ARGUMENT, msg() << "'" << key << "' must either be 'float16' or 'float32', not '"
                                     << value << "'");
}

// src/poplar_kge.cpp:144-152.  A power below 1 is no norm, and pow of a negative base needs an integer power.
void read_regulariser(const SettingMap& s, const std::string& prefix, float& power, float& weight) {
    power = get_float(s, prefix + ".power");
    weight = get_float(s, prefix + ".weight");
    if (weight < 0.f) fail(KGE_INVALID_ARGUMENT, msg() << "'" << prefix << ".weight' must not be negative");
    if (weight > 0.f && !(power >= 1.f))
        fail(KGE_INVALID_ARGUMENT, msg() << "'" << prefix << ".power' must be at least 1, actual: " << power);
}

}  // namespace

Config parse_config(const SettingMap& s) {
    Config c{};
    c.n_shard = get_unsigned(s, "model.n_shard");
    const std::string device = get_string(s, "execution.device");
    if (device != "cpu" && device != "ipu" && device != "ipu_model" && device != "cuda") {
        fail(KGE_INVALID_ARGUMENT, msg() << "Unexpected setting \"device\": '" << device
                                         << "', expected \"cuda\" (or the reference's \"cpu\" / \"ipu\")");
    }
    c.seed = get_unsigned(s, "model.seed");
    const std::string score_fn = get_string(s, "model.score_fn");
    const std::string distance_fn = get_string(s, "model.distance_fn");
    c.n_entity = get_unsigned(s, "model.n_entity");
    c.n_relation_type = get_unsigned(s, "model.n_relation_type");
    c.d = get_unsigned(s, "model.embedding_size");
    c.f = get_unsigned(s, "model.entity_feature_size");
    const unsigned mlp = get_unsigned(s, "model.feature_mlp_size");
    const float dropout = get_float(s, "model.feature_dropout");
    c.share_networks = get_bool(s, "model.share_feature_networks");
    c.gamma = get_float(s, "model.gamma");
    c.init_scale = get_float(s, "model.init_scale");
    c.beta_m = get_float(s, "training.adam_beta_m");
    c.beta_v = get_float(s, "training.adam_beta_v");
    c.epsilon = get_float(s, "training.adam_epsilon");
    c.weight_decay = get_float(s, "training.weight_decay");
    const std::string mod_prefix = "training.learning_rate_modifiers.";
    for (auto& kv : s) {
        if (kv.first.compare(0, mod_prefix.size(), mod_prefix) == 0) {
            c.lr_modifiers[kv.first.substr(mod_prefix.size())] = get_float(s, kv.first);
        }
    }
    c.batch_size = get_unsigned(s, "data.batch_size");
    c.a2a_size = get_unsigned(s, "data.a2a_size");
    c.adversarial_scale = get_float(s, "model.negative_adversarial_scale");
    const std::string loss = get_string(s, "training.loss.type");
    read_regulariser(s, "training.embedding_regularisation", c.reg_power[0], c.reg_weight[0]);
    read_regulariser(s, "training.feature_regularisation", c.reg_power[1], c.reg_weight[1]);
    read_regulariser(s, "training.hidden_regularisation", c.reg_power[2], c.reg_weight[2]);
    c.correction_weight = loss == "softmax" ? get_float(s, "training.loss.correction_weight") : 0.f;
    c.loss_scale = get_float(s, "training.loss_scale");
    c.n_step = get_unsigned(s, "execution.train_steps_per_program_run");
    c.rw_batch = get_unsigned(s, "execution.rw_batch_size");
    c.predict_hr = get_unsigned(s, "execution.predict_hr_batch_size");
    c.predict_tail_batch = get_unsigned(s, "execution.predict_tail_batch_size");
    c.predict_n_best = get_unsigned(s, "execution.predict_n_best");
    c.state_type = parse_storage("execution.dtype", get_string(s, "execution.dtype"));
    c.feature_type = s.count("execution.feature_dtype")
                         ? parse_storage("execution.feature_dtype", get_string(s, "execution.feature_dtype"))
                         : c.state_type;
    c.value_bf16 = false;
    if (s.count("execution.value_dtype")) {
        const std::string v = get_string(s, "execution.value_dtype");
        if (v == "bfloat16") c.value_bf16 = true;
        else if (v != "float32" && v != "float16")
            fail(KGE_INVALID_ARGUMENT, msg() << "'execution.value_dtype' must be 'bfloat16' or the row type, not '" << v << "'");
        if (c.value_bf16 && c.state_type != ST_F32)
            fail(KGE_INVALID_ARGUMENT, "'execution.value_dtype' 'bfloat16' needs 'execution.dtype' 'float32' (the optimiser state stays float32)");
    }
    c.device_ordinal = get_or<unsigned>(s, "execution.device_ordinal", get_unsigned, 0u);
    c.rank = get_or<unsigned>(s, "execution.rank", get_unsigned, 0u);
    c.world = get_or<unsigned>(s, "execution.world_size", get_unsigned, 1u);
    c.cuda_graph = get_or<bool>(s, "execution.cuda_graph", get_bool, true);
    c.tensor_cores = get_or<bool>(s, "execution.tensor_cores", get_bool, true);
    c.l2_contraction = get_or<bool>(s, "execution.l2_contraction", get_bool, false);

    if (score_fn == "TransE") c.score_fn = SCORE_TRANSE;
    else if (score_fn == "DistMult") c.score_fn = SCORE_DISTMULT;
    else if (score_fn == "ComplEx") c.score_fn = SCORE_COMPLEX;
    else if (score_fn == "RotatE") c.score_fn = SCORE_ROTATE;
    else if (score_fn == "TransH") c.score_fn = SCORE_TRANSH;
    else
        fail(KGE_INVALID_ARGUMENT, msg() << "'model.score_fn' must be one of 'TransE', 'ComplEx', 'RotatE', "
                                            "'TransH', or 'DistMult', not '" << score_fn << "'");
    if (distance_fn == "L1" || distance_fn == "L1_old") c.dist_fn = DIST_L1;
    else if (distance_fn == "L2" || distance_fn == "L2_old") c.dist_fn = DIST_L2;
    else if (distance_fn == "MatMul") c.dist_fn = DIST_DOT;
    else
        fail(KGE_INVALID_ARGUMENT, msg() << "'model.distance_fn' must be one of 'L1', 'L1_old', 'L2', 'L2_old' "
                                            "or 'MatMul', not '" << distance_fn << "'");
    // TransH's score is the L1 form whatever the setting says (src/poplar_kge.cpp:552-565)
    if (c.score_fn == SCORE_TRANSH) c.dist_fn = DIST_L1;
    if (loss == "logsigmoid") c.loss_fn = LOSS_LOGSIGMOID;
    else if (loss == "softmax") c.loss_fn = LOSS_SOFTMAX;
    else
        fail(KGE_INVALID_ARGUMENT, msg() << "'training.loss.type' must be one of 'logsigmoid' or 'softmax', not '"
                                         << loss << "'");
    c.mlp = mlp;
    if (!(dropout >= 0.f && dropout < 1.f)) fail(KGE_INVALID_ARGUMENT, msg() << "'model.feature_dropout' must be in [0, 1), actual: " << dropout);
    c.dropout = dropout;
    if (c.state_type == ST_F16 && c.feature_type != ST_F16)
        fail(KGE_INVALID_ARGUMENT, "'execution.feature_dtype' must be 'float16' when 'execution.dtype' is 'float16'");

    // Parameters are sliced by rows over the shards (src/poplar_kge.cpp:294-300).
    auto divisible = [&](const char* name, unsigned rows, unsigned cols) {
        if (rows % c.n_shard)
            fail(KGE_INVALID_ARGUMENT, msg() << "Parameter '" << name << "' shape[0] (" << rows
                                             << ") is not divisible by n_shard (" << c.n_shard
                                             << "). Note shape: (" << rows << ", " << cols << ")");
    };
    if (c.n_shard == 0 || c.world == 0 || c.n_shard % c.world || c.rank >= c.world)
        fail(KGE_INVALID_ARGUMENT, msg() << "n_shard (" << c.n_shard << ") must be a positive multiple of "
                                            "execution.world_size (" << c.world << ") and rank < world_size");
    divisible("relation_embedding", c.n_relation_type, c.d);
    if (c.f) divisible(c.share_networks ? "feature_projection" : "head_feature_projection", c.f, c.d);
    if (c.f && c.mlp) {  // src/poplar_kge.cpp:260-265
        divisible(c.share_networks ? "mlp_up_projection" : "head_mlp_up_projection", 2 * c.d, c.mlp);
        divisible(c.share_networks ? "mlp_down_projection" : "head_mlp_down_projection", c.mlp, c.d);
    }
    for (auto& kv : c.lr_modifiers) {
        const bool known = kv.first == "entity_embedding" || kv.first == "relation_embedding" ||
                           (c.score_fn == SCORE_TRANSH && kv.first == "relation_normal") ||
                           (c.mlp && c.f && c.share_networks && (kv.first == "mlp_up_projection" || kv.first == "mlp_down_projection")) ||
                           (c.mlp && c.f && !c.share_networks &&
                            (kv.first == "head_mlp_up_projection" || kv.first == "head_mlp_down_projection" ||
                             kv.first == "tail_mlp_up_projection" || kv.first == "tail_mlp_down_projection")) ||
                           (c.share_networks ? kv.first == "feature_projection"
                                             : (kv.first == "head_feature_projection" ||
                                                kv.first == "tail_feature_projection"));
        if (!known)
            fail(KGE_INVALID_ARGUMENT, msg() << "Bad training.learning_rate_modifier: unknown parameter '"
                                             << kv.first << "'");
    }
    if (c.d == 0 || c.batch_size == 0 || c.a2a_size == 0 || c.n_step == 0 || c.n_entity == 0)
        fail(KGE_INVALID_ARGUMENT, "embedding_size, batch_size, a2a_size, n_entity and "
                                   "train_steps_per_program_run must be positive");
    if ((c.score_fn == SCORE_COMPLEX || c.score_fn == SCORE_ROTATE) && (c.d & 1))
        fail(KGE_INVALID_ARGUMENT, "ComplEx and RotatE need an even 'model.embedding_size'");
    if (c.score_fn == SCORE_ROTATE && c.dist_fn == DIST_DOT)
        fail(KGE_INVALID_ARGUMENT, "RotatE scores by a distance: 'model.distance_fn' must be 'L1' or 'L2'");
    if (c.score_fn == SCORE_TRANSH && c.d >= UINT32_MAX / kMaxSortItems)
        fail(KGE_INVALID_ARGUMENT, msg() << "TransH: 'model.embedding_size' is limited to " << UINT32_MAX / kMaxSortItems - 1);
    if (c.n_tail() < 2) fail(KGE_INVALID_ARGUMENT, "n_shard * a2a_size must be at least 2");
    if ((size_t)c.batch_size + c.n_tail() > (size_t)kMaxSortItems)
        fail(KGE_INVALID_ARGUMENT, msg() << "batch_size + n_shard * a2a_size (" << c.n_remote()
                                         << ") exceeds this engine's limit of " << kMaxSortItems);
    return c;
}

// ---------------------------------------------------------------------------
// Dispatch over the row storage types.

#define KGE_DISPATCH_ROW(cfg, ...)                                          \
    do {                                                                     \
        if ((cfg).state_type == ST_F32 && (cfg).feature_type == ST_F32) {    \
            using ST = float; using FT = float; __VA_ARGS__;                 \
        } else if ((cfg).state_type == ST_F32) {                             \
            using ST = float; using FT = __half; __VA_ARGS__;                \
        } else {                                                             \
            using ST = __half; using FT = __half; __VA_ARGS__;               \
        }                                                                    \
    } while (0)

namespace {
size_t type_bytes(int storage) { return storage == ST_F32 ? 4 : 2; }
unsigned ceil_div(unsigned a, unsigned b) { return (a + b - 1) / b; }
}  // namespace

// ---------------------------------------------------------------------------
// Construction

void* Engine::device_alloc(size_t bytes) {
    void* p = nullptr;
    KGE_CUDA(cudaMalloc(&p, std::max<size_t>(bytes, 16)));
    allocations_.push_back(p);
    return p;
}

size_t Engine::arena_offset_dense(int which) const {
    const size_t flags = round_up(sizeof(unsigned) * kFlagWords, 256);
    return flags + (size_t)which * round_up(n_dense_ * sizeof(float), 256);
}
size_t Engine::arena_offset_shard(unsigned local, int which) const {
    // per local shard: tails | grad_recv | lower plane of tails
    const size_t row_block = round_up((size_t)cfg_.n_tail() * cfg_.d * sizeof(float), 256);
    const size_t per_shard = 3 * row_block;
    const size_t base = arena_offset_dense(4) + (size_t)local * per_shard;
    return base + (size_t)which * row_block;
}
// Receive buffer of the partial dense gradients: one slot of `dense_chunk_` floats per shard of the job.
size_t Engine::arena_offset_dense_recv() const { return arena_offset_predict(3); }
size_t Engine::arena_offset_predict(int which) const {
    // gathered queries [n_shard, hr, D] | result scores | result rows, each [n_local, n_shard, hr, n_best]
    // (TransH: the predicted tails, then the unit normals, src/poplar_kge.cpp:823-828)
    const size_t queries = round_up((size_t)(cfg_.score_fn == SCORE_TRANSH ? 2 : 1) * cfg_.n_shard * cfg_.predict_hr * cfg_.d * sizeof(float), 256);
    const size_t results = round_up((size_t)n_local_ * cfg_.n_shard * cfg_.predict_hr * cfg_.predict_n_best * 4, 256);
    const size_t base = arena_offset_shard(n_local_, 0);
    return base + (which == 0 ? 0 : which == 1 ? queries : which == 2 ? queries + results : queries + 2 * results);
}
size_t Engine::arena_size() const {
    return arena_offset_dense_recv() + round_up((size_t)cfg_.n_shard * dense_chunk_ * sizeof(float), 256);
}

Engine::Engine(const SettingMap& settings) : cfg_(parse_config(settings)) {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || (int)cfg_.device_ordinal >= count) {
        cudaGetLastError();
        fail(KGE_RUNTIME_ERROR, msg() << "Could not attach to CUDA device " << cfg_.device_ordinal << " ("
                                      << count << " visible)");
    }
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    n_local_ = cfg_.n_shard / cfg_.world;
    shard0_ = cfg_.rank * n_local_;

    const size_t sb = type_bytes(cfg_.state_type), fb = type_bytes(cfg_.feature_type);
    const uint32_t seg = (uint32_t)round_up(cfg_.d * sb, 16), value_seg = cfg_.value_bf16 ? (uint32_t)round_up(cfg_.d * 2, 16) : seg;
    layout_.off_m = value_seg;
    layout_.off_q = value_seg + seg;
    layout_.off_feat = value_seg + 2 * seg;
    layout_.row_bytes = layout_.off_feat + (uint32_t)round_up(cfg_.f * fb, 16);
    layout_.value_bf16 = cfg_.value_bf16 ? 1u : 0u;
    layout_.d = cfg_.d;
    layout_.f = cfg_.f;

    adam_.beta_m = cfg_.beta_m;
    adam_.beta_v = cfg_.beta_v;
    adam_.one_minus_beta_m = 1.0f - cfg_.beta_m;
    adam_.one_minus_beta_v = 1.0f - cfg_.beta_v;
    adam_.epsilon = cfg_.epsilon;
    adam_.weight_decay = cfg_.weight_decay;

    // dense vector: relation table | projection(s)
    proj_elems_ = (size_t)cfg_.f * cfg_.d;
    dense_bounds_[0] = 0;
    dense_bounds_[1] = (size_t)cfg_.n_relation_type * cfg_.d;
    dense_bounds_[2] = dense_bounds_[1] + (cfg_.n_net() >= 1 ? proj_elems_ : 0);
    dense_bounds_[3] = dense_bounds_[2] + (cfg_.n_net() >= 2 ? proj_elems_ : 0);
    dense_bounds_[4] = dense_bounds_[3] + (cfg_.score_fn == SCORE_TRANSH ? (size_t)cfg_.n_relation_type * cfg_.d : 0);
    for (unsigned net = 0; net < 2; ++net) {  // the feature MLP's projections: up [2D, M], down [M, D]
        const bool present = cfg_.mlp > 0 && net < cfg_.n_net();
        dense_bounds_[5 + 2 * net] = dense_bounds_[4 + 2 * net] + (present ? (size_t)2 * cfg_.d * cfg_.mlp : 0);
        dense_bounds_[6 + 2 * net] = dense_bounds_[5 + 2 * net] + (present ? (size_t)cfg_.mlp * cfg_.d : 0);
    }
    n_dense_ = dense_bounds_[kDenseParams];
    auto modifier = [&](const std::string& name) {
        auto it = cfg_.lr_modifiers.find(name);
        return it == cfg_.lr_modifiers.end() ? 1.0f : it->second;
    };
    entity_lr_mod_ = modifier("entity_embedding");
    dense_lr_mod_[0] = modifier("relation_embedding");
    std::vector<std::string> proj_names;
    if (cfg_.n_net() == 1) proj_names = {"feature_projection"};
    if (cfg_.n_net() == 2) proj_names = {"head_feature_projection", "tail_feature_projection"};
    // With no features the reference still declares an empty projection; it is listed with
    // shape [0, D] and carries no data.
    if (cfg_.n_net() == 0)
        proj_names = cfg_.share_networks
                         ? std::vector<std::string>{"feature_projection"}
                         : std::vector<std::string>{"head_feature_projection", "tail_feature_projection"};
    for (size_t i = 0; i < proj_names.size() && i < 2; ++i) dense_lr_mod_[1 + i] = modifier(proj_names[i]);

    auto add_variable = [&](const std::string& name, size_t rows, size_t cols, size_t offset, bool flat = false) {
        const char* suffix[3] = {"", "/adam_m", "/adam_v"};
        for (int k = 0; k < 3; ++k)
            variables_.push_back({name + suffix[k], KGE_F32, {rows, cols}, offset, k, flat});
    };
    // RotatE's relations are angles, one per complex pair (src/poplar_kge.cpp:248-251); the table keeps
    // rows of d floats all the same and uses their first half
    add_variable("relation_embedding", cfg_.n_relation_type, cfg_.score_fn == SCORE_ROTATE ? cfg_.d / 2 : cfg_.d, 0);
    for (size_t i = 0; i < proj_names.size(); ++i)
        add_variable(proj_names[i], cfg_.f, cfg_.d, cfg_.f ? dense_bounds_[1 + i] : n_dense_);
    if (cfg_.score_fn == SCORE_TRANSH) {  // src/poplar_kge.cpp:252-255
        add_variable("relation_normal", cfg_.n_relation_type, cfg_.d, dense_bounds_[3]);
        dense_lr_mod_[3] = modifier("relation_normal");
    }
    if (cfg_.mlp > 0 && cfg_.n_net() > 0)
        for (unsigned net = 0; net < cfg_.n_net(); ++net) {
            const std::string prefix = proj_names[net].substr(0, proj_names[net].size() - std::string("feature_projection").size());
            add_variable(prefix + "mlp_up_projection", 2 * cfg_.d, cfg_.mlp, dense_bounds_[4 + 2 * net], true);
            add_variable(prefix + "mlp_down_projection", cfg_.mlp, cfg_.d, dense_bounds_[5 + 2 * net]);
            dense_lr_mod_[4 + 2 * net] = modifier(prefix + "mlp_up_projection");
            dense_lr_mod_[5 + 2 * net] = modifier(prefix + "mlp_down_projection");
        }
    variables_.push_back({"step", KGE_U32, {cfg_.n_shard}, 0, 3, false});

    // Every process owns (reduces and updates) an equal share of the rows of the dense vector, dealt
    // out in turn: row r belongs to process r % world, as its row r / world.
    const size_t dense_rows = cfg_.n_relation_type + (size_t)cfg_.n_net() * cfg_.f + (cfg_.score_fn == SCORE_TRANSH ? cfg_.n_relation_type : 0) +
                              (cfg_.mlp > 0 ? (size_t)cfg_.n_net() * 3 * cfg_.mlp : 0);
    dense_chunk_rows_ = std::max<size_t>(1, (dense_rows + cfg_.world - 1) / cfg_.world);
    dense_chunk_ = dense_chunk_rows_ * cfg_.d;
    own_rows_ = dense_rows > cfg_.rank ? (dense_rows - cfg_.rank + cfg_.world - 1) / cfg_.world : 0;

    const unsigned tiles = ceil_div(cfg_.f, 64) * ceil_div(cfg_.d, 64) * std::max(1u, cfg_.n_net());
    proj_splits_ = (int)std::min(8u, std::max(1u, ceil_div(148, std::max(1u, tiles))));
    proj_rows_per_split_ = (int)round_up(ceil_div(cfg_.n_remote(), proj_splits_), 32);

    KGE_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    KGE_CUDA(cudaStreamCreateWithFlags(&side_stream_, cudaStreamNonBlocking));
    if (const char* v = std::getenv("KGE_SPLIT_POPULAR_ROWS")) split_popular_rows_ = std::atoi(v) != 0;
    // Worth its launch only where other processes wait for the shard that holds the popular entity:
    // measured 85.0 against 82.9 us per step on one GPU, where nobody waits.
    heavy_route_ = cfg_.world >= 4;
    if (const char* v = std::getenv("KGE_ROUTE_POPULAR_ROWS")) heavy_route_ = std::atoi(v) != 0;
    if (const char* v = std::getenv("KGE_FUSE_DENSE_UPDATE")) fuse_dense_env_ = std::atoi(v) != 0;
    if (const char* v = std::getenv("KGE_PREDICT_FILTER_IN_SCORES")) filter_in_scores_ = std::atoi(v) != 0;
    // Which work runs beside the step's chain: bit 0 the relation gradients, bit 1 the next step's gather.
    side_streams_ = 3u;
    if (const char* v = std::getenv("KGE_SIDE_STREAMS")) side_streams_ = (unsigned)std::atoi(v) & 3u;
    KGE_CUDA(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
    if (n_local_ > 1 && cfg_.world == 1) {
        ev_shard_.resize(n_local_, nullptr);
        for (cudaEvent_t& e : ev_shard_) KGE_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    for (cudaEvent_t& e : ev_join_) KGE_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (RunEvents& r : ev_runs_)
        for (cudaEvent_t* e : {&r.begin, &r.end, &r.stage[0], &r.stage[1]}) KGE_CUDA(cudaEventCreate(e));
    // The step of batched launches: rows of 16 bytes, which its contractions' operands need, and lookups of a block of hidden
    // rows that fit its staging area.  Scores and coefficients get rows of a multiple of eight, so that any batch will do.
    planes_ = cfg_.tensor_cores && cfg_.d % 4 == 0 && cfg_.n_remote() <= (unsigned)tc::kRouteMaxLookups;
    if (const char* v = std::getenv("KGE_PLANE_CONTRACTIONS")) planes_ = planes_ && std::atoi(v) != 0;
    if (mlp_on()) planes_ = false;  // the MLP sits between the projection and the lookups: the step of separate kernels
    score_ld_ = planes_ ? (unsigned)round_up(cfg_.n_tail(), 8) : cfg_.n_tail();
    // Without features a hidden row is the stored value: the lookups read the table itself and, but for the regularisers, which
    // take the hidden rows and the state of a gathered copy, so does the row update.
    table_lookups_ = planes_ && cfg_.f == 0;
    direct_rows_ = table_lookups_ && !cfg_.regularised();
    // Shards of one launch.  With several processes the hand-over counters count the blocks of one shard's kernel at a time.
    group_ = cfg_.world == 1 ? std::min(n_local_, (unsigned)kShardBatch) : 1u;
    branches_ = cfg_.world > 1 ? 1u : planes_ ? ceil_div(n_local_, group_) : n_local_;
    alone_ = branches_ == 1;
    // Where every shard is in every launch no gradient has to wait for another launch: the projection gradient's
    // contraction (over all shards' rows) and the relation rows' blocks of the entity update apply the Adam step
    // themselves and k_dense_update is not launched.
    fuse_dense_ = fuse_dense_env_ && planes_ && cfg_.world == 1 && cfg_.n_shard <= (unsigned)kShardBatch;
    // fp16 features are widened into rows of their own; the lower plane of fp32 features keeps the
    // stride of the rows whose feature part is its upper plane (one stride per operand)
    bf16_planes_ = planes_ && cfg_.value_bf16 && cfg_.dist_fn == DIST_DOT && cfg_.score_fn != SCORE_TRANSH && cfg_.d % 8 == 0 && cfg_.n_tail() % 8 == 0 && cfg_.batch_size % 8 == 0 &&
                   (cfg_.a2a_size * cfg_.d) % 2 == 0;
    feat_stride_ = cfg_.feature_type == ST_F16 ? (uint32_t)round_up(cfg_.f, 4) : layout_.row_bytes / 4;
    allocate();
    peer_arena_.assign(cfg_.world, nullptr);
    peer_arena_[cfg_.rank] = arena_;
    if (cfg_.world == 1) {
        build_pointer_tables();
        connected_ = true;
    }
}

Engine::~Engine() {
    cudaSetDevice((int)cfg_.device_ordinal);
    if (stream_) cudaStreamSynchronize(stream_);
    for (StepGraph& g : graphs_) if (g.exec) cudaGraphExecDestroy(g.exec);
    for (cudaEvent_t e : event_pool_) cudaEventDestroy(e);
    for (unsigned p = 0; p < peer_arena_.size(); ++p)
        if (p != cfg_.rank && peer_arena_[p]) cudaIpcCloseMemHandle(peer_arena_[p]);
    for (void* p : allocations_) cudaFree(p);
    for (cudaEvent_t e : ev_io_) if (e) cudaEventDestroy(e);
    if (pinned_) cudaFreeHost(pinned_);
    for (const RunEvents& r : ev_runs_)
        for (cudaEvent_t e : {r.begin, r.end, r.stage[0], r.stage[1]}) if (e) cudaEventDestroy(e);
    if (ev_fork_) cudaEventDestroy(ev_fork_);
    for (cudaEvent_t e : ev_join_) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : ev_shard_) if (e) cudaEventDestroy(e);
    if (side_stream_) cudaStreamDestroy(side_stream_);
    if (stream_) cudaStreamDestroy(stream_);
}

void Engine::allocate() {
    const unsigned B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote(), D = cfg_.d;
    const bool two_nets = cfg_.n_net() == 2;
    const bool multiplicative = cfg_.score_fn != SCORE_TRANSE;

    arena_ = (uint8_t*)device_alloc(arena_size());
    KGE_CUDA(cudaMemset(arena_, 0, arena_size()));
    dense_ = (float*)(arena_ + arena_offset_dense(0));
    dense_m_ = (float*)(arena_ + arena_offset_dense(1));
    dense_v_ = (float*)(arena_ + arena_offset_dense(2));
    dense_lo_ = (float*)(arena_ + arena_offset_dense(3));

    shards_.resize(n_local_);
    table_stride_ = round_up((size_t)cfg_.n_entity * layout_.row_bytes, 256);
    uint8_t* tables = (uint8_t*)device_alloc(n_local_ * table_stride_);
    KGE_CUDA(cudaMemset(tables, 0, n_local_ * table_stride_));
    const size_t score_elems = (size_t)B * score_ld_;
    // what the projection's gradient contracts over lies shard behind shard, one operand for all of them
    uint8_t* rows_all[2] = {nullptr, nullptr};
    float *wide_all[2] = {nullptr, nullptr}, *lo_all[2] = {nullptr, nullptr}, *d_hid_all[2] = {nullptr, nullptr}, *d_hid_lo_all[2] = {nullptr, nullptr};
    for (int i = 0; i < 2; ++i) {
        if (!direct_rows_) rows_all[i] = (uint8_t*)device_alloc((size_t)n_local_ * R * layout_.row_bytes);
        if (planes_ && cfg_.f) (cfg_.feature_type == ST_F16 ? wide_all : lo_all)[i] = (float*)device_alloc((size_t)n_local_ * R * feat_stride_ * 4);
        if (i == 1 && !two_nets) continue;
        d_hid_all[i] = (float*)device_alloc((size_t)n_local_ * R * D * 4);
        if (planes_ && cfg_.f) d_hid_lo_all[i] = (float*)device_alloc((size_t)n_local_ * R * D * 4);
    }
    for (unsigned l = 0; l < n_local_; ++l) {
        ShardBuffers& b = shards_[l];
        b.table = tables + l * table_stride_;
        for (int i = 0; i < 2; ++i) {
            if (rows_all[i]) b.rows_c2[i] = rows_all[i] + (size_t)l * R * layout_.row_bytes;
            if (wide_all[i]) b.feat_wide2[i] = wide_all[i] + (size_t)l * R * feat_stride_;
            if (lo_all[i]) b.feat_lo2[i] = lo_all[i] + (size_t)l * R * feat_stride_;
        }
        b.d_hid_h = d_hid_all[0] + (size_t)l * R * D;
        if (d_hid_all[1]) b.d_hid_t = d_hid_all[1] + (size_t)l * R * D;
        if (d_hid_lo_all[0]) b.d_hid_h_lo = d_hid_lo_all[0] + (size_t)l * R * D;
        if (d_hid_lo_all[1]) b.d_hid_t_lo = d_hid_lo_all[1] + (size_t)l * R * D;
        b.hid_h = (float*)device_alloc((size_t)R * D * 4);
        b.hid_t = two_nets || dropout_on() ? (float*)device_alloc((size_t)R * D * 4) : b.hid_h;  // dropout: each call has its own mask
        b.pred = (float*)device_alloc((size_t)B * D * 4);
        b.raw = (float*)device_alloc(score_elems * 4);
        b.coeff = (float*)device_alloc(score_elems * 4);
        b.d_pred = (float*)device_alloc((size_t)B * D * 4);
        b.d_head = multiplicative ? (float*)device_alloc((size_t)B * D * 4) : b.d_pred;
        b.d_relrow = multiplicative ? (float*)device_alloc((size_t)B * D * 4) : b.d_pred;
        if (mlp_on()) {
            const size_t M = cfg_.mlp;
            for (unsigned net = 0; net < cfg_.n_net(); ++net) {
                b.mlp_cat[net] = (float*)device_alloc((size_t)R * 2 * D * 4);
                b.mlp_pre[net] = (float*)device_alloc((size_t)R * M * 4);
            }
            b.mlp_out = (float*)device_alloc((size_t)R * D * 4);
            b.mlp_d_pre = (float*)device_alloc((size_t)R * M * 4);
            b.mlp_d_cat = (float*)device_alloc((size_t)R * 2 * D * 4);
            b.d_val = (float*)device_alloc((size_t)R * D * 4);
            b.mlp_dw_up = (float*)device_alloc((size_t)2 * D * M * 4);
            b.mlp_dw_down = (float*)device_alloc((size_t)M * D * 4);
        }
        if (cfg_.score_fn == SCORE_TRANSH) {
            b.nrm = (float*)device_alloc((size_t)B * D * 4);
            b.d_nrm = (float*)device_alloc((size_t)B * D * 4);
            b.d_normrow = (float*)device_alloc((size_t)B * D * 4);
            b.pair_s = (float*)device_alloc(score_elems * 4);
            b.pair_u = (float*)device_alloc(score_elems * 4);
            // (what lies behind a row's last column is multiplied with coefficients of zero)
            KGE_CUDA(cudaMemset(b.pair_s, 0, score_elems * 4));
            KGE_CUDA(cudaMemset(b.pair_u, 0, score_elems * 4));
        }
        if (cfg_.regularised()) {
            b.reg_val = (float*)device_alloc((size_t)R * D * 4);
            b.reg_h = (float*)device_alloc((size_t)R * D * 4);
            b.reg_t = two_nets || dropout_on() ? (float*)device_alloc((size_t)R * D * 4) : nullptr;
            b.reg_loss_rows = (float*)device_alloc((size_t)R * 4);
        }
        b.proj_partial = (float*)device_alloc(std::max<size_t>(1, cfg_.n_net()) * proj_splits_ * proj_elems_ * 4);
        b.loss_rows = (float*)device_alloc((size_t)B * 4);
        b.tails = (float*)(arena_ + arena_offset_shard(l, 0));
        b.grad_recv = (float*)(arena_ + arena_offset_shard(l, 1));
        b.dense_partial = (float*)(arena_ + arena_offset_dense_recv()) + (size_t)(shard0_ + l) * dense_chunk_;
        b.dense_dst = (float**)device_alloc(sizeof(float*) * cfg_.world);
        b.heavy_partial = (float*)device_alloc((size_t)kHeavySlots * 2 * D * 4);
        b.heavy_counter = (unsigned*)device_alloc(kHeavySlots * sizeof(unsigned));
        KGE_CUDA(cudaMemset(b.heavy_counter, 0, kHeavySlots * sizeof(unsigned)));
        b.send_dst = (float**)device_alloc(sizeof(float*) * cfg_.n_shard);
        b.grad_dst = (float**)device_alloc(sizeof(float*) * cfg_.n_shard);
        b.send_lo_dst = (float**)device_alloc(sizeof(float*) * cfg_.n_shard);
        b.tails_lo = (float*)(arena_ + arena_offset_shard(l, 2));
        if (planes_) {
            b.pred_lo = (float*)device_alloc((size_t)B * D * 4);
            b.coeff_lo = (float*)device_alloc(score_elems * 4);
        }
        b.predict_score_dst = (float**)device_alloc(sizeof(float*) * cfg_.n_shard);
        b.predict_index_dst = (uint32_t**)device_alloc(sizeof(uint32_t*) * cfg_.n_shard);
    }
    d_epoch_ = (unsigned*)device_alloc(sizeof(unsigned));
    d_xchg_words_ = (unsigned*)device_alloc(2 * XCHG_KINDS * sizeof(unsigned));
    KGE_CUDA(cudaMemset(d_xchg_words_, 0, 2 * XCHG_KINDS * sizeof(unsigned)));
    if (const char* on = std::getenv("KGE_EXCHANGE_TRACE"); on && on[0] && on[0] != '0') {
        const size_t bytes = (size_t)kTraceSlots * XCHG_KINDS * 3 * sizeof(unsigned long long);
        d_xchg_trace_ = (unsigned long long*)device_alloc(bytes);
        KGE_CUDA(cudaMemset(d_xchg_trace_, 0, bytes));
    }
    KGE_CUDA(cudaMemset(d_epoch_, 0, sizeof(unsigned)));
    {
        // room for the two problems of the largest paired launch, kTcMaxSplits partial tiles each
        const size_t per_problem = std::max<size_t>({(size_t)R * D, (size_t)(std::max(B, T)) * D, (size_t)cfg_.f * D, (size_t)B * T});
        tc_ws_floats_ = per_problem * kTcMaxSplits;
        tc_ws_ = (float*)device_alloc(2 * tc_ws_floats_ * 4);
        tc_ws_rowsum_ = (float*)device_alloc(2 * (size_t)kTcMaxSplits * std::max(B, T) * 4);
    }
    d_peer_flags_ = (unsigned**)device_alloc(sizeof(unsigned*) * cfg_.world);
    d_partials_ = (const float**)device_alloc(sizeof(float*) * cfg_.n_shard);
    d_replicas_ = (float**)device_alloc(sizeof(float*) * cfg_.world);
    d_replicas_lo_ = (float**)device_alloc(sizeof(float*) * cfg_.world);

    const size_t steps = (size_t)n_local_ * cfg_.n_step;
    {
        size_t at = 0;
        const size_t stream_words[5] = {steps * R, steps * T, steps * B, steps * B, steps * B};
        for (int i = 0; i < 5; ++i) stage_at_[i] = at, at += round_up(stream_words[i], 4);
        keys_at_ = at;
        sizes_at_ = keys_at_ + cfg_.n_step;
        loss_at_ = sizes_at_ + cfg_.n_step;
        status_at_ = loss_at_ + n_local_;
        run_words_ = status_at_ + 3;
        d_run_ = (uint32_t*)device_alloc(run_words_ * 4);
        KGE_CUDA(cudaMemset(d_run_ + loss_at_, 0, (run_words_ - loss_at_) * 4));
        KGE_CUDA(cudaMallocHost((void**)&pinned_, run_words_ * 4));
    }
    d_remote_ = d_run_ + stage_at_[0];
    d_a2a_ = d_run_ + stage_at_[1];
    d_head_ = d_run_ + stage_at_[2];
    d_relation_ = d_run_ + stage_at_[3];
    d_tail_ = d_run_ + stage_at_[4];
    d_step_key_ = d_run_ + keys_at_;
    d_step_size_ = reinterpret_cast<float*>(d_run_ + sizes_at_);
    d_loss_total_ = reinterpret_cast<float*>(d_run_ + loss_at_);
    d_tc_status_ = d_run_ + status_at_;
    d_status_ = d_tc_status_ + 1;
    d_planes_short_ = d_tc_status_ + 2;
    d_ent_perm_ = (uint32_t*)device_alloc(steps * (B + T) * 4);
    d_ent_off_ = (uint32_t*)device_alloc(steps * (R + 1) * 4);
    d_rel_perm_ = (uint32_t*)device_alloc(steps * B * 4);
    d_rel_off_ = (uint32_t*)device_alloc(steps * (cfg_.n_relation_type + 1) * 4);
    d_first_slot_ = (uint32_t*)device_alloc(steps * R * 4);
    if (table_lookups_) d_lookup_row_ = (uint32_t*)device_alloc(steps * (B + T) * 4);
    d_heavy_parts_ = (uint4*)device_alloc(steps * kHeavySlots * sizeof(uint4));
    d_row_info_ = (uint4*)device_alloc(steps * 2 * R * sizeof(uint4));
    d_heavy_count_ = (uint32_t*)device_alloc(steps * 4);
    KGE_CUDA(cudaMemset(d_heavy_count_, 0, steps * 4));
    d_loss_last_ = (float*)device_alloc(n_local_ * 4);
    d_loss_counter_ = (unsigned*)device_alloc(n_local_ * sizeof(unsigned));
    KGE_CUDA(cudaMemset(d_loss_counter_, 0, n_local_ * sizeof(unsigned)));
    if (cfg_.regularised()) {
        d_reg_loss_ = (float*)device_alloc(n_local_ * 2 * sizeof(float));
        KGE_CUDA(cudaMemset(d_reg_loss_, 0, n_local_ * 2 * sizeof(float)));
        d_reg_counter_ = (unsigned*)device_alloc(n_local_ * sizeof(unsigned));
        KGE_CUDA(cudaMemset(d_reg_counter_, 0, n_local_ * sizeof(unsigned)));
    }

    const size_t rw = (size_t)n_local_ * cfg_.rw_batch;
    d_rw_idx_ = (uint32_t*)device_alloc(std::max<size_t>(rw, (size_t)n_local_ * cfg_.predict_hr * 2) * 4);
    KGE_CUDA(cudaDeviceSynchronize());
}

void Engine::build_pointer_tables() {
    const size_t block = (size_t)cfg_.a2a_size * cfg_.d;  // floats per (src, dst) block
    std::vector<float*> send(cfg_.n_shard), grad(cfg_.n_shard), send_lo(cfg_.n_shard);
    std::vector<const float*> partials(cfg_.n_shard);
    for (unsigned l = 0; l < n_local_; ++l) {
        const unsigned me = shard0_ + l;
        for (unsigned d = 0; d < cfg_.n_shard; ++d) {
            const unsigned owner = d / n_local_, dl = d % n_local_;
            uint8_t* base = peer_arena_[owner];
            send[d] = (float*)(base + arena_offset_shard(dl, 0)) + (size_t)me * block;
            grad[d] = (float*)(base + arena_offset_shard(dl, 1)) + (size_t)me * block;
            // the companion plane holds rows of D bf16 values (half a float each) in the bf16 tier
            send_lo[d] = (float*)(base + arena_offset_shard(dl, 2)) + (size_t)me * block / (bf16_planes_ ? 2 : 1);
        }
        KGE_CUDA(cudaMemcpy(shards_[l].send_lo_dst, send_lo.data(), sizeof(float*) * cfg_.n_shard, cudaMemcpyHostToDevice));
        KGE_CUDA(cudaMemcpy(shards_[l].send_dst, send.data(), sizeof(float*) * cfg_.n_shard, cudaMemcpyHostToDevice));
        KGE_CUDA(cudaMemcpy(shards_[l].grad_dst, grad.data(), sizeof(float*) * cfg_.n_shard, cudaMemcpyHostToDevice));
        // predict: results of tail shard `me` for the queries of shard d land in d's [d_local][me] block
        std::vector<float*> pscore(cfg_.n_shard);
        std::vector<uint32_t*> pindex(cfg_.n_shard);
        const size_t result_block = (size_t)cfg_.predict_hr * cfg_.predict_n_best;
        for (unsigned d = 0; d < cfg_.n_shard; ++d) {
            uint8_t* base = peer_arena_[d / n_local_];
            const size_t slot = ((size_t)(d % n_local_) * cfg_.n_shard + me) * result_block;
            pscore[d] = (float*)(base + arena_offset_predict(1)) + slot;
            pindex[d] = (uint32_t*)(base + arena_offset_predict(2)) + slot;
        }
        KGE_CUDA(cudaMemcpy(shards_[l].predict_score_dst, pscore.data(), sizeof(float*) * cfg_.n_shard, cudaMemcpyHostToDevice));
        KGE_CUDA(cudaMemcpy(shards_[l].predict_index_dst, pindex.data(), sizeof(uint32_t*) * cfg_.n_shard, cudaMemcpyHostToDevice));
    }
    for (unsigned l = 0; l < n_local_; ++l) {
        // where shard shard0_ + l writes its partial dense gradient: its slot in every owner's receive buffer
        std::vector<float*> dst(cfg_.world);
        for (unsigned p = 0; p < cfg_.world; ++p)
            dst[p] = (float*)(peer_arena_[p] + arena_offset_dense_recv()) + (size_t)(shard0_ + l) * dense_chunk_;
        KGE_CUDA(cudaMemcpy(shards_[l].dense_dst, dst.data(), sizeof(float*) * cfg_.world, cudaMemcpyHostToDevice));
    }
    for (unsigned d = 0; d < cfg_.n_shard; ++d)
        partials[d] = (const float*)(arena_ + arena_offset_dense_recv()) + (size_t)d * dense_chunk_;
    KGE_CUDA(cudaMemcpy(d_partials_, partials.data(), sizeof(float*) * cfg_.n_shard, cudaMemcpyHostToDevice));
    std::vector<float*> replicas(cfg_.world), replicas_lo(cfg_.world);
    std::vector<unsigned*> flags(cfg_.world);
    for (unsigned p = 0; p < cfg_.world; ++p) {
        replicas[p] = (float*)(peer_arena_[p] + arena_offset_dense(0));
        replicas_lo[p] = (float*)(peer_arena_[p] + arena_offset_dense(3));
        flags[p] = (unsigned*)(peer_arena_[p] + arena_offset_flags());
    }
    KGE_CUDA(cudaMemcpy(d_replicas_, replicas.data(), sizeof(float*) * cfg_.world, cudaMemcpyHostToDevice));
    KGE_CUDA(cudaMemcpy(d_replicas_lo_, replicas_lo.data(), sizeof(float*) * cfg_.world, cudaMemcpyHostToDevice));
    KGE_CUDA(cudaMemcpy(d_peer_flags_, flags.data(), sizeof(unsigned*) * cfg_.world, cudaMemcpyHostToDevice));
}

// ---------------------------------------------------------------------------
// Multi-process set-up

namespace {
struct CommHandle {
    cudaIpcMemHandle_t mem;
    uint32_t rank, world;
    uint64_t arena_bytes;
};
}  // namespace

size_t Engine::comm_handle_bytes() { return sizeof(CommHandle); }

void Engine::comm_export(void* out) const {
    CommHandle h{};
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    KGE_CUDA(cudaIpcGetMemHandle(&h.mem, arena_));
    h.rank = cfg_.rank;
    h.world = cfg_.world;
    h.arena_bytes = arena_size();
    std::memcpy(out, &h, sizeof(h));
}

void Engine::comm_connect(const void* handles, size_t world) {
    if (world != cfg_.world)
        fail(KGE_INVALID_ARGUMENT, msg() << "kge_comm_connect: got " << world << " handles, world_size is " << cfg_.world);
    if (connected_) fail(KGE_LOGIC_ERROR, "kge_comm_connect: already connected");
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    const CommHandle* all = static_cast<const CommHandle*>(handles);
    for (unsigned p = 0; p < cfg_.world; ++p) {
        CommHandle h;
        std::memcpy(&h, all + p, sizeof(h));
        if (h.rank != p || h.world != cfg_.world || h.arena_bytes != arena_size())
            fail(KGE_INVALID_ARGUMENT, msg() << "kge_comm_connect: handle " << p << " does not match this engine's settings");
        if (p == cfg_.rank) continue;
        void* ptr = nullptr;
        cudaError_t err = cudaIpcOpenMemHandle(&ptr, h.mem, cudaIpcMemLazyEnablePeerAccess);
        if (err != cudaSuccess) {
            cudaGetLastError();
            fail(KGE_RUNTIME_ERROR, msg() << "Could not attach to the device memory of rank " << p << ": "
                                          << cudaGetErrorString(err));
        }
        peer_arena_[p] = (uint8_t*)ptr;
    }
    build_pointer_tables();
    connected_ = true;
}

// ---------------------------------------------------------------------------
// Host array checks (src/poplar_kge.cpp:69-106)

namespace {
const char* dtype_name(int dtype) {
    return dtype == KGE_F32 ? "float" : dtype == KGE_U32 ? "unsigned int" : "half";
}
std::string shape_string(const std::vector<size_t>& shape) {
    msg m;
    m << "(";
    for (size_t i = 0; i < shape.size(); ++i) m << (i ? ", " : "") << shape[i];
    m << ")";
    return m;
}
}  // namespace

HostArray& Engine::find_array(std::vector<HostArray>& arrays, const std::string& name, int dtype,
                              const std::vector<size_t>& shape) {
    for (HostArray& a : arrays) {
        if (a.name != name) continue;
        if (a.dtype != dtype)
            fail(KGE_INVALID_ARGUMENT, msg() << "'" << name << "' expected array of type " << dtype_name(dtype)
                                             << ", actual: " << dtype_name(a.dtype));
        if (a.shape != shape)
            fail(KGE_INVALID_ARGUMENT, msg() << "'" << name << "' expected array of shape " << shape_string(shape)
                                             << ", actual: " << shape_string(a.shape));
        if (!a.data && a.count()) fail(KGE_INVALID_ARGUMENT, msg() << "'" << name << "' has a null data pointer");
        return a;
    }
    fail(KGE_INVALID_ARGUMENT, msg() << "Key not found '" << name << "'");
}

// ---------------------------------------------------------------------------
// Commands

void Engine::run(const std::string& command, std::vector<HostArray>& arrays, const std::string& variable) {
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    if (command == "train_step_loop") return cmd_train_step_loop(arrays);
    if (command == "predict") return cmd_predict(arrays);
    if (command == "read_entity") return cmd_read_entity(arrays);
    if (command == "write_entity") return cmd_write_entity(arrays, false);
    if (command == "write_entity_rows") return cmd_write_entity(arrays, true);
    if (command == "read_entity_range") return cmd_entity_range(arrays, true);
    if (command == "write_entity_range") return cmd_entity_range(arrays, false);
    if (command == "initialise_entities") return cmd_initialise_entities();
    if (command == "entity_layout") {
        // `layout` u32 [4]: bytes of a stored row, rows per shard, local shards, the first local shard
        HostArray& out = find_array(arrays, "layout", KGE_U32, {4});
        uint32_t* o = static_cast<uint32_t*>(out.data);
        o[0] = layout_.row_bytes, o[1] = (uint32_t)cfg_.n_entity, o[2] = (uint32_t)n_local_, o[3] = (uint32_t)(cfg_.rank * n_local_);
        return;
    }
    if (command == "dump_entity_rows") return cmd_copy_entity_range(arrays, true);
    if (command == "restore_entity_rows") return cmd_copy_entity_range(arrays, false);
    if (command == "load_triples") return cmd_load_triples(arrays);
    if (command == "sample_batch") return cmd_sample_batch(arrays, false);
    if (command == "train_step_loop_sampled") return cmd_sample_batch(arrays, true);
    if (command == "read" || command == "write") return cmd_read_write_variable(arrays, variable, command == "write");
    fail(KGE_INVALID_ARGUMENT, msg() << "Unknown command '" << command << "'");
}

void Engine::cmd_train_step_loop(std::vector<HostArray>& arrays) {
    HostArray& lr = find_array(arrays, "learning_rate", KGE_F32, {n_local_});
    HostArray& loss = find_array(arrays, "loss", KGE_F32, {n_local_});
    stage_batch(arrays, static_cast<const float*>(lr.data));
    train_staged(static_cast<const float*>(lr.data)[0], static_cast<float*>(loss.data));
}

// The words of the coming run that change with it: Adam step sizes (src/fructose/frnn.cpp:42-59, in fp32), the steps'
// numbers, and zeros for the loss totals.
void Engine::write_run_words(float learning_rate) {
    uint32_t* keys = pinned_ + keys_at_;
    float* sizes = reinterpret_cast<float*>(pinned_ + sizes_at_);
    for (unsigned i = 0; i < cfg_.n_step; ++i) {
        const float t = (float)(step_ + 1 + i);
        keys[i] = (uint32_t)(step_ + 1 + i);
        sizes[i] = (std::sqrt(1.0f - std::pow(cfg_.beta_v, t)) / (1.0f - std::pow(cfg_.beta_m, t))) * learning_rate;
    }
    std::memset(pinned_ + loss_at_, 0, n_local_ * 4);
}

void Engine::stage_batch(std::vector<HostArray>& arrays, const float* learning_rate) {
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    const size_t n = n_local_, S = cfg_.n_step, B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote();
    HostArray& remote = find_array(arrays, "remote", KGE_U32, {n, S, R});
    HostArray& a2a = find_array(arrays, "a2a", KGE_U32, {n, S, cfg_.n_shard, cfg_.a2a_size});
    HostArray& head = find_array(arrays, "head", KGE_U32, {n, S, B});
    HostArray& relation = find_array(arrays, "relation", KGE_U32, {n, S, B});
    HostArray& tail = find_array(arrays, "tail", KGE_U32, {n, S, B});
    // The reference would read out of bounds on a bad index; here it is refused on the host.
    auto check_below = [](const HostArray& a, uint32_t limit, const char* what) {
        const uint32_t* p = static_cast<const uint32_t*>(a.data);
        const size_t count = a.count();
        for (size_t i = 0; i < count; ++i)
            if (p[i] >= limit)
                fail(KGE_INVALID_ARGUMENT, msg() << "'" << a.name << "' holds index " << p[i] << " at position " << i
                                                 << ", which is not below " << what << " (" << limit << ")");
    };
    // One pass per stream copies into the pinned buffer and takes the maximum; only a stream with a bad index is
    // walked again for its position.  A batch that fails a check is not staged: the engine refuses to train until one
    // passes all five.
    staged_ = false;
    run_words_uploaded_ = false;
    if (uploads_pending_) KGE_CUDA(cudaStreamSynchronize(stream_));  // the pinned buffer may still be in flight
    uploads_pending_ = true;
    struct Upload { const HostArray* a; uint32_t limit; const char* what; };
    const Upload uploads[5] = {{&remote, cfg_.n_entity, "model.n_entity"}, {&a2a, (uint32_t)R, "the number of gathered rows"},
                               {&head, (uint32_t)R, "the number of gathered rows"}, {&relation, cfg_.n_relation_type, "model.n_relation_type"},
                               {&tail, (uint32_t)T, "n_shard * a2a_size"}};
    // Up to 256 KB one transfer carries everything, the run's words included (a transfer costs the host 3 us, the link
    // 1 us); above that each stream travels while the next one is copied and checked.
    const bool one_transfer = keys_at_ * 4 <= 256 * 1024;
    for (int i = 0; i < 5; ++i) {
        const Upload& u = uploads[i];
        uint32_t* out = pinned_ + stage_at_[i];
        const size_t count = u.a->count();
        if (copy_and_max(out, static_cast<const uint32_t*>(u.a->data), count) >= u.limit) check_below(*u.a, u.limit, u.what);
        if (!one_transfer) KGE_CUDA(cudaMemcpyAsync(d_run_ + stage_at_[i], out, count * 4, cudaMemcpyHostToDevice, stream_));
    }
    if (learning_rate) {
        write_run_words(*learning_rate);
        run_words_uploaded_ = true;
    }
    const size_t from = one_transfer ? 0 : keys_at_, to = learning_rate ? status_at_ : keys_at_;
    if (to > from) KGE_CUDA(cudaMemcpyAsync(d_run_ + from, pinned_ + from, (to - from) * 4, cudaMemcpyHostToDevice, stream_));
    prepare_staged();
}

// The sort-and-segment tables of the staged index streams (the backward of the row gather).
void Engine::prepare_staged() {
    const size_t n = n_local_, S = cfg_.n_step, B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote();
    KGE_CUDA(cudaEventRecord(ev_runs_[ev_run_].stage[0], stream_));
    k_prepare_segments<<<(unsigned)(n * S), 512, 0, stream_>>>(
        d_head_, d_a2a_, d_relation_, d_remote_, (int)B, (int)T, (int)R, (int)cfg_.n_relation_type, d_ent_perm_,
        d_ent_off_, d_rel_perm_, d_rel_off_, d_first_slot_, split_popular_rows_ ? d_heavy_parts_ : nullptr, d_heavy_count_, d_row_info_, d_lookup_row_);
    KGE_CUDA(cudaGetLastError());
    KGE_CUDA(cudaEventRecord(ev_runs_[ev_run_].stage[1], stream_));
    staged_ = true;
    stage_fresh_ = true;
}

// ---------------------------------------------------------------------------
// The batch sampler on the device (src/python/poplar_kge_dataset.py:199-263, 310-393)

// "load_triples": the training triples as local rows, sorted by (head shard, tail shard) bucket:
// `triples` u32 [3, n] (head row, relation, tail row), `bucket_offset` / `bucket_count` u32
// [n_shard, n_shard], `shard_to_count` u32 [n_shard] (real rows per shard).  All shards of the job,
// on every process: a shard's batch names positives that other shards' heads drew.
void Engine::cmd_load_triples(std::vector<HostArray>& arrays) {
    const size_t n = cfg_.n_shard;
    HostArray* triples = nullptr;
    for (HostArray& a : arrays)
        if (a.name == "triples") triples = &a;
    if (!triples) fail(KGE_INVALID_ARGUMENT, "Key not found 'triples'");
    if (triples->dtype != KGE_U32 || triples->shape.size() != 2 || triples->shape[0] != 3 || triples->shape[1] == 0)
        fail(KGE_INVALID_ARGUMENT, "'triples' expected an unsigned int array of shape (3, n_triples)");
    const size_t n_triples = triples->shape[1];
    HostArray& offset = find_array(arrays, "bucket_offset", KGE_U32, {n, n});
    HostArray& count = find_array(arrays, "bucket_count", KGE_U32, {n, n});
    HostArray& rows = find_array(arrays, "shard_to_count", KGE_U32, {n});
    const uint32_t *h_off = static_cast<const uint32_t*>(offset.data), *h_cnt = static_cast<const uint32_t*>(count.data);
    const uint32_t *h_rows = static_cast<const uint32_t*>(rows.data), *h_tri = static_cast<const uint32_t*>(triples->data);
    if (cfg_.batch_size % cfg_.n_shard || cfg_.a2a_size <= cfg_.batch_size / cfg_.n_shard)
        fail(KGE_INVALID_ARGUMENT, msg() << "Expected batch_size (" << cfg_.batch_size << ") to be a multiple of n_shard and a2a_size ("
                                         << cfg_.a2a_size << ") to be >= batch_size/n_shard");
    for (size_t b = 0; b < n * n; ++b) {
        if (h_cnt[b] == 0) fail(KGE_INVALID_ARGUMENT, msg() << "'bucket_count' has an empty (head shard, tail shard) bucket " << b);
        if ((size_t)h_off[b] + h_cnt[b] > n_triples) fail(KGE_INVALID_ARGUMENT, "'bucket_offset' + 'bucket_count' passes the end of 'triples'");
    }
    for (size_t s = 0; s < n; ++s)
        if (h_rows[s] == 0 || h_rows[s] >= cfg_.n_entity)
            fail(KGE_INVALID_ARGUMENT, msg() << "'shard_to_count' (" << h_rows[s] << ") must be between 1 and model.n_entity - 1");
    for (size_t i = 0; i < n_triples; ++i) {
        if (h_tri[i] >= cfg_.n_entity || h_tri[2 * n_triples + i] >= cfg_.n_entity || h_tri[i] == 0 || h_tri[2 * n_triples + i] == 0)
            fail(KGE_INVALID_ARGUMENT, msg() << "'triples' names a row outside [1, model.n_entity) at triple " << i);
        if (h_tri[n_triples + i] >= cfg_.n_relation_type)
            fail(KGE_INVALID_ARGUMENT, msg() << "'triples' names relation " << h_tri[n_triples + i] << " at triple " << i);
    }
    uint32_t* d_triples = (uint32_t*)device_alloc(3 * n_triples * 4);
    uint32_t* d_meta = (uint32_t*)device_alloc((2 * n * n + n) * 4);
    KGE_CUDA(cudaMemcpy(d_triples, h_tri, 3 * n_triples * 4, cudaMemcpyHostToDevice));
    KGE_CUDA(cudaMemcpy(d_meta, h_off, n * n * 4, cudaMemcpyHostToDevice));
    KGE_CUDA(cudaMemcpy(d_meta + n * n, h_cnt, n * n * 4, cudaMemcpyHostToDevice));
    KGE_CUDA(cudaMemcpy(d_meta + 2 * n * n, h_rows, n * 4, cudaMemcpyHostToDevice));
    sampler_ = SamplerData{d_triples, n_triples, d_meta, d_meta + n * n, d_meta + 2 * n * n};
}

void Engine::sample_and_stage(uint32_t seed) {
    if (!sampler_.triples) fail(KGE_LOGIC_ERROR, "no training triples: run \"load_triples\" first");
    k_sample_batch<<<(unsigned)(n_local_ * cfg_.n_step), 512, 0, stream_>>>(sampler_, seed, sample_run_++, (int)cfg_.n_shard, (int)shard0_,
                                                                             (int)cfg_.n_step, (int)cfg_.batch_size, (int)cfg_.a2a_size,
                                                                             d_remote_, d_a2a_, d_head_, d_relation_, d_tail_, cfg_.n_entity - 1);
    KGE_CUDA(cudaGetLastError());
    prepare_staged();
}

// "sample_batch": draws one program run's index streams on the device (`sample_seed` u32 [1]) and
// stages them; any of remote / a2a / head / relation / tail given (local shapes of
// "train_step_loop") receives a copy.  "train_step_loop_sampled": the same, then the steps:
// `learning_rate`, `loss` as for "train_step_loop"; no index array crosses the host.
void Engine::cmd_sample_batch(std::vector<HostArray>& arrays, bool train) {
    const size_t n = n_local_, S = cfg_.n_step, B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote();
    HostArray& seed = find_array(arrays, "sample_seed", KGE_U32, {1});
    HostArray *lr = nullptr, *loss = nullptr;
    if (train) {
        lr = &find_array(arrays, "learning_rate", KGE_F32, {n});
        loss = &find_array(arrays, "loss", KGE_F32, {n});
    }
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    run_words_uploaded_ = false;
    sample_and_stage(static_cast<const uint32_t*>(seed.data)[0]);
    struct Stream { const char* name; uint32_t* device; std::vector<size_t> shape; };
    const Stream streams[5] = {{"remote", d_remote_, {n, S, R}}, {"a2a", d_a2a_, {n, S, cfg_.n_shard, cfg_.a2a_size}},
                               {"head", d_head_, {n, S, B}}, {"relation", d_relation_, {n, S, B}}, {"tail", d_tail_, {n, S, B}}};
    for (const Stream& st : streams)
        for (HostArray& a : arrays)
            if (a.name == st.name) {
                HostArray& out = find_array(arrays, st.name, KGE_U32, st.shape);
                copy_out(out.data, st.device, out.count() * 4, out.count() * 4, 1);
            }
    if (train) train_staged(static_cast<const float*>(lr->data)[0], static_cast<float*>(loss->data));
}


void Engine::train_staged(float learning_rate, float* loss) {
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    require_usable();
    if (!staged_) fail(KGE_LOGIC_ERROR, "kge_train_staged called before kge_stage_batch");
    if (!connected_) fail(KGE_LOGIC_ERROR, "world_size > 1 but kge_comm_connect has not been called");
    if (!run_words_uploaded_) {
        if (uploads_pending_) KGE_CUDA(cudaStreamSynchronize(stream_));
        uploads_pending_ = true;
        write_run_words(learning_rate);
        KGE_CUDA(cudaMemcpyAsync(d_run_ + keys_at_, pinned_ + keys_at_, (status_at_ - keys_at_) * 4, cudaMemcpyHostToDevice, stream_));
    }
    run_words_uploaded_ = false;
    std::optional<ShardStreams> streams;
    steps_queued_ = false;
    try {
        KGE_CUDA(cudaEventRecord(ev_runs_[ev_run_].begin, stream_));
        if (cfg_.cuda_graph && !kernel_timing_ && launched_before_) {
            launch_step_graphs();
        } else {
            launched_before_ = true;
            launch_counter_ = 0;
            if (kernel_timing_) {
                // hold the stream while the host queues the run, so the event pairs bracket kernels only
                k_delay<<<1, 1, 0, stream_>>>(20ll * 1000 * 1000);
                KGE_CUDA(cudaGetLastError());
            }
            streams.emplace(*this);
            steps_queued_ = true;
            launch_steps(0, cfg_.n_step);
            last_launches_ = launch_counter_;
        }
        KGE_CUDA(cudaEventRecord(ev_runs_[ev_run_].end, stream_));
        // the loss totals and the status words are neighbours: one transfer brings both
        KGE_CUDA(cudaMemcpyAsync(pinned_ + loss_at_, d_run_ + loss_at_, (run_words_ - loss_at_) * 4, cudaMemcpyDeviceToHost, stream_));
        KGE_CUDA(cudaStreamSynchronize(stream_));
    } catch (...) {
        // some of the steps have moved the rows, and the step counter has not followed
        if (steps_queued_) unusable_ = "an earlier program run failed after some of its steps: this engine's state is between two runs and it must be rebuilt";
        throw;
    }
    if (streams) streams->give_back();
    uploads_pending_ = false;
    ms_pending_ = true;
    // the sort-and-segment preparation belongs to the step (it is the backward of the row
    // gather): its device time counts towards the first run of a staged batch
    ms_counts_stage_ = stage_fresh_;
    stage_fresh_ = false;
    ev_run_ ^= 1;
    timing_collect();
    step_ += cfg_.n_step;
    raise_device_status(pinned_ + status_at_);
    const float* host_loss = reinterpret_cast<const float*>(pinned_ + loss_at_);
    if (loss)
        for (unsigned l = 0; l < n_local_; ++l) loss[l] = host_loss[l] / (float)cfg_.n_step;
}

// Both status words come back in one copy (they are neighbours in device memory).  A wait that gave
// up leaves this engine's kernels out of step with the other processes' (their hand-over epochs
// disagree from then on), so the engine refuses further device commands: it must be rebuilt.
void Engine::check_device_status() {
    KGE_CUDA(cudaMemcpyAsync(pinned_ + status_at_, d_tc_status_, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, stream_));
    KGE_CUDA(cudaStreamSynchronize(stream_));
    raise_device_status(pinned_ + status_at_);
}
void Engine::raise_device_status(const unsigned* words) {
    const unsigned status[2] = {words[0], words[1]};  // [0] the tensor-core pipeline, [1] the hand-overs between processes
    if (!status[0] && !status[1]) return;
    unusable_ = "a device-side wait of an earlier command gave up: this engine is out of step with the other processes and must be rebuilt";
    KGE_CUDA(cudaMemset(d_tc_status_, 0, sizeof(status)));
    if (status[0]) fail(KGE_DEVICE_STATUS, msg() << "a bounded wait on the tensor-core pipeline gave up (code " << status[0] << ")");
    fail(KGE_DEVICE_STATUS, msg() << "a device-side wait for rank " << (status[1] - 1)
                                  << " gave up: that process did not reach the same step");
}

void Engine::require_usable() const {
    if (unusable_) fail(KGE_LOGIC_ERROR, unusable_);
}

void Engine::set_kernel_timing(bool on) {
    kernel_timing_ = on;
    if (on) kernel_times_.clear();
}

size_t Engine::kernel_time_count() const { return kernel_times_.size(); }

void Engine::kernel_time(size_t index, const char** name, float* ms, unsigned long long* launches) const {
    if (index >= kernel_times_.size()) fail(KGE_INVALID_ARGUMENT, "kge_kernel_time: index past the end");
    auto it = kernel_times_.begin();
    std::advance(it, index);
    if (name) *name = it->first.c_str();
    if (ms) *ms = it->second.ms;
    if (launches) *launches = it->second.launches;
}

void Engine::last_run_stats(float* ms, unsigned long long* launches) const {
    if (ms_pending_) {
        const RunEvents& run = ev_runs_[ev_run_ ^ 1];
        KGE_CUDA(cudaEventElapsedTime(&last_ms_, run.begin, run.end));
        if (ms_counts_stage_) {
            float stage_ms = 0.f;
            KGE_CUDA(cudaEventElapsedTime(&stage_ms, run.stage[0], run.stage[1]));
            last_ms_ += stage_ms;
        }
        ms_pending_ = false;
    }
    if (ms) *ms = last_ms_;
    if (launches) *launches = last_launches_;
}

// Wraps one kernel launch: counts it and, when per-kernel timing is on, brackets it with a
// pair of events on the engine's stream.
#define KGE_LAUNCH(name, ...)            \
    do {                                 \
        timing_begin(name);              \
        __VA_ARGS__;                     \
        timing_end();                    \
        ++launch_counter_;               \
    } while (0)

bool dependent_launch_enabled() {
    static const bool enabled = [] {
        const char* off = std::getenv("KGE_NO_DEPENDENT_LAUNCH");
        return !(off && off[0] && off[0] != '0');
    }();
    return enabled;
}

namespace {
// Streams for the shards' branches, lent out while steps are queued or captured (Engine::ShardStreams): making one costs the host about 2 ms,
// as much as capturing a short run.  At most kKept per device wait for the next borrower; the rest are destroyed.
class StreamPool {
   public:
    static StreamPool& instance() {
        static StreamPool* pool = new StreamPool;  // never destroyed: CUDA may be gone before static destructors run
        return *pool;
    }
    cudaStream_t take() {
        const int slot = current_device_slot();
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (slot >= 0 && !free_[slot].empty()) {
                cudaStream_t st = free_[slot].back();
                free_[slot].pop_back();
                return st;
            }
        }
        cudaStream_t st = nullptr;
        KGE_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        return st;
    }
    void give(cudaStream_t st) {
        const int slot = current_device_slot();
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (slot >= 0 && free_[slot].size() < kKept) {
                free_[slot].push_back(st);
                return;
            }
        }
        cudaStreamDestroy(st);  // work still queued on it completes first
    }

   private:
    static constexpr size_t kKept = 16;
    std::mutex mutex_;
    std::vector<cudaStream_t> free_[kMaxDeviceOrdinals];
};
}  // namespace

// The shards' streams, from before the first step is queued until the streams are out of the capture that recorded the
// steps, or until the steps themselves are over: StreamPool serves every engine of the process, and an engine on another
// thread may borrow a stream the moment it is back.  After an error they are destroyed, not lent again.
Engine::ShardStreams::ShardStreams(Engine& e) : engine_(e) {
    if (e.branches_ < 2 || e.kernel_timing_) return;
    e.shard_streams_.assign(e.branches_, nullptr);
    for (unsigned l = 1; l < e.branches_; ++l) e.shard_streams_[l] = StreamPool::instance().take();
}
void Engine::ShardStreams::give_back() {
    for (cudaStream_t st : engine_.shard_streams_)
        if (st) StreamPool::instance().give(st);
    engine_.shard_streams_.clear();
}
Engine::ShardStreams::~ShardStreams() {
    for (cudaStream_t st : engine_.shard_streams_)
        if (st) cudaStreamDestroy(st);
    engine_.shard_streams_.clear();
}

// A program run as a short chain of CUDA graphs, each four times as long as the one before: on the run that makes them,
// every graph but the first (a single step) is captured and instantiated while its predecessor runs on the GPU.  That is
// an engine's second run; the first goes out as plain launches, at about 3 us of host time each, while a graph costs 12 us
// per kernel in a chain and up to 22 us among the branches of several shards (capture 1, instantiation 9 to 19, upload 2).
// Milliseconds of an engine's first / second / later run, graphs made in the first and in the second (with a stream per shard),
// and now that the shards share launches:
//   demo preset, 5 steps of 2 shards   1.45 / 0.31 / 0.29    0.58 / 1.46 / 0.29    0.25 / 0.73 / 0.19
//   4 shards of TransE-L1, 20 steps    13.8 / 1.95 / 1.91    2.75 / 13.1 / 1.92    1.37 / 1.54 / 1.26
//   2 shards of the headline, 20       7.36 / 3.66 / 2.98    4.26 / 7.14 / 3.00    2.34 / 3.71 / 2.22
//   headline model, 100 steps          16.9 / 8.36 / 7.79    9.08 / 15.4 / 7.80    7.53 / 14.6 / 7.21
void Engine::launch_step_graphs() {
    if (graphs_.empty()) {
        unsigned length = 1;
        for (unsigned first = 0; first < cfg_.n_step; first += length, length *= 4)
            graphs_.push_back({first, std::min(first + length, cfg_.n_step), nullptr, 0});
        // a last graph shorter than its predecessor's launch joins it
        if (graphs_.size() > 1 && graphs_.back().end - graphs_.back().first < (graphs_.back().first - graphs_[graphs_.size() - 2].first) / 2) {
            graphs_[graphs_.size() - 2].end = cfg_.n_step;
            graphs_.pop_back();
        }
    }
    last_launches_ = 0;
    for (StepGraph& g : graphs_) {
        if (!g.exec && !record_graph(g)) {  // no room for it: the rest of this run goes out kernel by kernel
            steps_queued_ = true;
            launch_counter_ = 0;
            launch_steps(g.first, cfg_.n_step);
            last_launches_ += launch_counter_;
            return;
        }
        KGE_CUDA(cudaGraphLaunch(g.exec, stream_));
        steps_queued_ = true;
        last_launches_ += g.launches;
    }
}

// Captures and instantiates the steps of `g`; false where the driver has no memory for the graph.
bool Engine::record_graph(StepGraph& g) {
    cudaGraph_t graph = nullptr;
    launch_counter_ = 0;
    {
        ShardStreams streams(*this);
        KGE_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
        try {
            launch_steps(g.first, g.end);
        } catch (...) {
            cudaStreamEndCapture(stream_, &graph);
            if (graph) cudaGraphDestroy(graph);
            throw;
        }
        KGE_CUDA(cudaStreamEndCapture(stream_, &graph));
        streams.give_back();
    }
    const cudaError_t err = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    g.launches = launch_counter_;
    if (err == cudaSuccess) return true;
    g.exec = nullptr;
    if (err != cudaErrorMemoryAllocation) KGE_CUDA(err);
    cudaGetLastError();
    return false;
}

void Engine::launch_steps(unsigned first, unsigned end) {
    if (first == 0) launch_gather(0, stream_);
    for (unsigned step = first; step < end; ++step) launch_one_step(step);
    if (end < cfg_.n_step) return;
    // The last kernel of a step only publishes its dense parameters.  The run ends when every
    // process's share has arrived in this process's copy (values and optimiser state), so that a
    // "read" or "predict" issued straight after the run sees the finished step without a host barrier.
    launch_exchange_wait(XCHG_DENSE_PARAMS);
}

// The step's rows, gathered into the compact copy every later kernel of the step reads (two
// copies, for even and odd steps).  The gather of step s + 1 needs only the rows step s has
// updated, so it runs beside the projection gradient and the dense update of step s.
void Engine::launch_gather(unsigned step, cudaStream_t stream) {
    for (unsigned l = 0; l < n_local_; l += group_) launch_gather(step, l, std::min(group_, n_local_ - l), stream);
}
void Engine::launch_gather(unsigned step, unsigned l0, unsigned n, cudaStream_t stream) {
    if (direct_rows_) return;
    const unsigned R = cfg_.n_remote();
    ShardArgs<GatherArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        shards.s[i] = GatherArgs{b.table, d_remote_ + ((size_t)(l0 + i) * cfg_.n_step + step) * R, b.rows_c2[step & 1], feature_planes(b, step & 1)};
    }
    KGE_LAUNCH("gather", KGE_CUDA(launch_dependent(k_gather_step_rows, dim3(ceil_div(R, 8), n), dim3(256), 0, stream, shards, layout_.row_bytes, (int)R)));
}

FeaturePlanes Engine::feature_planes(const ShardBuffers& b, unsigned parity) const {
    FeaturePlanes fp{};
    fp.wide = b.feat_wide2[parity];
    fp.lo = b.feat_lo2[parity];
    fp.stride = feat_stride_;
    fp.off_feat = layout_.off_feat;
    return fp;
}

// Fork: what is launched on the returned stream starts after everything queued on the main stream
// so far.  While per-kernel timing is on, everything stays on the main stream.
cudaStream_t Engine::side_begin() {
    if (kernel_timing_ || !side_streams_) return stream_;
    KGE_CUDA(cudaEventRecord(ev_fork_, stream_));
    KGE_CUDA(cudaStreamWaitEvent(side_stream_, ev_fork_, 0));
    return side_stream_;
}
// ... the side work is complete here ...
void Engine::side_end(int which) {
    if (kernel_timing_ || !side_streams_) return;
    KGE_CUDA(cudaEventRecord(ev_join_[which], side_stream_));
}
// ... and the main stream waits for it here.
void Engine::side_join(int which) {
    if (kernel_timing_ || !side_streams_) return;
    KGE_CUDA(cudaStreamWaitEvent(stream_, ev_join_[which], 0));
}

// More local shards than a launch takes, or the step of separate kernels: the launches of a phase (hidden rows and lookups;
// scores and their gradients; row updates and projection gradient) work on a group of shards, or one shard, each and meet
// only at the exchange, so every branch of a phase is queued on a stream of its own (graph branches under capture).  The
// kernels of a step are short and mostly far too small to fill 148 SMs: side by side they take little longer than one of
// them.  us a step, groups of four one after the other -> side by side: sixteen shards of the demo's size 148 -> 62, eight of
// 256 x 512 x 100 L1 scores 122 -> 109, eight of 512 x 768 with features 401 -> 366, eight of TransH at that size 792 -> 707.
// Only with one process: the hand-over counters between processes count the blocks of one kernel at a time.
void Engine::shards_fork() {
    if (!shards_beside()) return;
    KGE_CUDA(cudaEventRecord(ev_fork_, stream_));
    for (unsigned l = 1; l < branches_; ++l) KGE_CUDA(cudaStreamWaitEvent(shard_streams_[l], ev_fork_, 0));
}
void Engine::shards_join() {
    if (!shards_beside()) return;
    for (unsigned l = 1; l < branches_; ++l) {
        KGE_CUDA(cudaEventRecord(ev_shard_[l], shard_streams_[l]));
        KGE_CUDA(cudaStreamWaitEvent(stream_, ev_shard_[l], 0));
    }
}

void Engine::launch_barrier() {
    if (cfg_.world == 1) return;
    BarrierArgs a;
    a.peer_flags = d_peer_flags_;
    a.my_epoch = d_epoch_;
    a.status = d_status_;
    a.rank = (int)cfg_.rank;
    a.world = (int)cfg_.world;
    a.max_spins = 2ull * 1000 * 1000;  // a second or two of 64 ns naps plus load latency
    KGE_LAUNCH("barrier", KGE_CUDA(launch_dependent(k_barrier, dim3(1), dim3(64), 0, stream_, a)));
    KGE_CUDA(cudaGetLastError());
}

// What the step's kernels need to publish and await the hand-overs between processes; with one
// process the kernels skip both.
ExchangeSync Engine::exchange_sync() const {
    ExchangeSync s{};
    s.peer_flags = d_peer_flags_;
    s.epochs = d_xchg_words_;
    s.counters = d_xchg_words_ + XCHG_KINDS;
    s.status = d_status_;
    s.rank = (int)cfg_.rank;
    s.world = (int)cfg_.world;
    s.max_spins = 1u << 28;
    s.timeout_ns = 2000ull * 1000ull * 1000ull;  // two seconds
    s.trace = d_xchg_trace_;
    return s;
}

void Engine::launch_exchange_wait(int kind) {
    if (cfg_.world == 1) return;
    KGE_LAUNCH("exchange_wait", KGE_CUDA(launch_dependent(k_exchange_wait, dim3(1), dim3(kMaxProcesses), 0, stream_, exchange_sync(), kind)));
}

void Engine::launch_exchange_signal(int kind) {
    if (cfg_.world == 1) return;
    KGE_LAUNCH("exchange_signal", KGE_CUDA(launch_dependent(k_exchange_signal, dim3(1), dim3(kMaxProcesses), 0, stream_, exchange_sync(), kind)));
}

void Engine::timing_begin(const char* name) {
    if (!kernel_timing_ || timed_.size() >= kMaxTimedLaunches) return;
    while (event_pool_.size() < 2 * (timed_.size() + 1)) {
        cudaEvent_t e = nullptr;
        KGE_CUDA(cudaEventCreate(&e));
        event_pool_.push_back(e);
    }
    timed_.push_back({name, event_pool_[2 * timed_.size()], event_pool_[2 * timed_.size() + 1]});
    timing_open_ = true;
    KGE_CUDA(cudaEventRecord(timed_.back().start, stream_));
}

void Engine::timing_end() {
    if (!timing_open_) return;
    timing_open_ = false;
    KGE_CUDA(cudaEventRecord(timed_.back().stop, stream_));
}

void Engine::timing_collect() {
    for (TimedLaunch& t : timed_) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, t.start, t.stop) == cudaSuccess) {
            KernelTime& k = kernel_times_[t.name];
            k.ms += ms;
            k.launches += 1;
        }
    }
    timed_.clear();
}

// How many k splits fill the GPU: about one block per SM, at least two 32-deep slices per split.
int Engine::tc_splits(unsigned tiles, unsigned k) const {
    const unsigned by_sms = std::max(1u, 148u / std::max(1u, tiles));
    const unsigned by_k = std::max(1u, k / 64u);
    int splits = (int)std::min<unsigned>({by_sms, by_k, (unsigned)kTcMaxSplits});
    // the splits of a tile run as one cluster: all tiles' clusters should be resident together
    while (splits > 1 && (unsigned)tc::max_resident_clusters(splits) < tiles) --splits;
    return splits;
}

// One launch for one or two contractions of the same kind (see tc_gemm.cuh).  With splits > 1
// the k range is divided and the partial tiles are reduced inside the kernel, in split order.
void Engine::launch_tc(const char* name, tc::GemmArgs* problems, int n_problems, int splits, bool a_exact, bool rowsum,
                       int wait_kind, int signal_kind) {
    for (int i = 0; i < n_problems; ++i) {
        tc::GemmArgs& g = problems[i];
        g.status = d_tc_status_;
        const unsigned tiles = ceil_div((unsigned)g.M, 128) * ceil_div((unsigned)g.N, 64);
        if (splits > 1 && tiles <= 4096 && (size_t)g.M * g.N * splits <= tc_ws_floats_) {
            g.k_per_split = (int)round_up(ceil_div((unsigned)g.K, (unsigned)splits), 32);
            g.ws = tc_ws_ + (size_t)i * tc_ws_floats_;
            g.ws_rowsum = tc_ws_rowsum_ + (size_t)i * kTcMaxSplits * std::max(cfg_.batch_size, cfg_.n_tail());
        } else {
            g.k_per_split = std::max(32, (int)round_up((unsigned)g.K, 32));
            g.ws = nullptr;
        }
    }
    if (!problems[0].ws || (n_problems > 1 && !problems[1].ws)) {
        splits = 1;
        for (int i = 0; i < n_problems; ++i) {
            problems[i].ws = nullptr;
            problems[i].k_per_split = std::max(32, (int)round_up((unsigned)problems[i].K, 32));
        }
    }
    cudaError_t err;
    timing_begin(name);
    int n_launches = 1;
    const ExchangeSync sync = exchange_sync();
    if (a_exact) err = rowsum ? tc::launch_pair<64, true, true>(problems, n_problems, splits, stream_, &n_launches, sync, wait_kind, signal_kind)
                              : tc::launch_pair<64, true, false>(problems, n_problems, splits, stream_, &n_launches, sync, wait_kind, signal_kind);
    else err = rowsum ? tc::launch_pair<64, false, true>(problems, n_problems, splits, stream_, &n_launches, sync, wait_kind, signal_kind)
                      : tc::launch_pair<64, false, false>(problems, n_problems, splits, stream_, &n_launches, sync, wait_kind, signal_kind);
    timing_end();
    launch_counter_ += (unsigned long long)n_launches;
    KGE_CUDA(err);
}

// How the k ranges of a launch's problems are divided over the blocks of clusters of `cluster` blocks: every problem over all
// of them or, where the launch allows it, over the divisor with which its blocks have the fewest slices to add up while all
// clusters are on the GPU at once.  Returns the longest chain of slices, 0 where the clusters do not fit.
static unsigned divide_k(const tc::PlaneProblem* problems, int n_problems, unsigned cluster, unsigned tile_n, unsigned slice, bool mixed, int* splits) {
    auto slices = [&](int i, unsigned s) { return std::max(1u, ceil_div(ceil_div((unsigned)problems[i].g.K, slice), s)); };
    unsigned tiles_n = 1;
    for (int i = 0; i < n_problems; ++i) tiles_n = std::max(tiles_n, ceil_div((unsigned)problems[i].g.N, tile_n));
    auto clusters = [&] {
        unsigned n = 0;
        for (int i = 0; i < n_problems; ++i) n += ceil_div(ceil_div((unsigned)problems[i].g.M, 128u), cluster / (unsigned)splits[i]) * tiles_n;
        return n;
    };
    const unsigned room = cluster > 1 ? (unsigned)tc::max_resident_plane_clusters((int)cluster) : ~0u;
    for (int i = 0; i < n_problems; ++i) splits[i] = mixed ? 1 : (int)cluster;
    if (clusters() > room) return 0;
    // divide the problem with the longest chain further while there is room for the blocks that takes
    for (bool further = mixed; further;) {
        int longest = 0;
        for (int i = 1; i < n_problems; ++i)
            if (slices(i, (unsigned)splits[i]) > slices(longest, (unsigned)splits[longest])) longest = i;
        int next = splits[longest] + 1;
        while (next <= (int)cluster && cluster % (unsigned)next) ++next;
        further = next <= (int)cluster;
        if (!further) break;
        const int before = splits[longest];
        splits[longest] = next;
        if (clusters() > room) splits[longest] = before, further = false;
    }
    unsigned chain = 0;
    for (int i = 0; i < n_problems; ++i) chain = std::max(chain, slices(i, (unsigned)splits[i]));
    return chain;
}

// One launch of the plane-fed contraction for problems of the same shape class, those of several local shards.  Tiles
// are 128 x 128 (128 x 64 for narrow outputs); the k range is divided over the blocks of a cluster so that about one block
// per SM is busy and every split keeps at least two slices.  The two score gradients of a batch with many more tails than
// triples have k ranges of very different length, and only the longer one wants dividing: with one number of splits for
// both, 256 x 1536 x 256 gradients walked 12 slices where 6 do (RotatE 82.9 -> 77.6 us a step).  Gradients from bfloat16
// operands stay with one number: their slices are short, the operands' way from L2 bounds them, and 1024 x 2048 x 512 with 16
// slices a block in place of 32 took 2 us longer.
void Engine::launch_planes(const char* name, tc::PlaneProblem* problems, int n_problems, int side, int wait_kind, int signal_kind,
                           const tc::Routing* routing) {
    int max_n = 0, max_k = 0;
    unsigned tiles = 0;
    bool alike = true;
    for (int i = 0; i < n_problems; ++i) {
        max_n = std::max(max_n, problems[i].g.N);
        alike = alike && problems[i].g.epilogue == problems[0].g.epilogue;
    }
    const bool half = problems[0].A.elem_bytes == 16;  // float16 planes: whole tiles of 128 x 128 (launch_prepared)
    const int tile_n = max_n > 64 || half ? 128 : 64;
    for (int i = 0; i < n_problems; ++i) {
        tiles += ceil_div((unsigned)problems[i].g.M, 128) * ceil_div((unsigned)max_n, (unsigned)tile_n);
        max_k = std::max(max_k, problems[i].g.K);
    }
    const unsigned slice = problems[0].A.elem_bytes == 2 || half ? 64u : 32u;  // slices of 16-bit operands are 64 deep
    int splits = (int)std::min<unsigned>({std::max(1u, 148u / std::max(1u, tiles)), std::max(1u, (unsigned)max_k / 64u),
                                          (unsigned)tc::kMaxClusterSplits});
    while (splits > 1 && (unsigned)tc::max_resident_plane_clusters(splits) < tiles) --splits;
    if (half) splits = 1;
    int each[tc::kMaxPlaneProblems];
    unsigned chain = divide_k(problems, n_problems, (unsigned)splits, (unsigned)tile_n, slice, false, each);
    if (n_problems > 1 && alike && problems[0].A.elem_bytes != 2 && tc::mixed_splits_allowed(side, problems[0].g.epilogue, tile_n)) {
        // worth it from two slices less on (a cluster's exchange where there was none costs about as much)
        for (unsigned cluster = 2; cluster <= (unsigned)tc::kMaxClusterSplits; cluster *= 2) {
            int other[tc::kMaxPlaneProblems];
            const unsigned c = divide_k(problems, n_problems, cluster, (unsigned)tile_n, slice, true, other);
            if (c == 0 || c + 2 > chain) continue;
            chain = c;
            splits = (int)cluster;
            std::copy(other, other + n_problems, each);
        }
    }
    for (int i = 0; i < n_problems; ++i) {
        tc::GemmArgs& g = problems[i].g;
        g.status = d_tc_status_;
        g.cluster_splits = each[i];
        g.k_per_split = (int)std::max<size_t>(slice, round_up(ceil_div((unsigned)g.K, (unsigned)each[i]), slice));
    }
    timing_begin(name);
    cudaError_t err;
    if (side == tc::SIDE_ROWSUM) err = tc::launch_planes<tc::SIDE_ROWSUM>(problems, n_problems, splits, tile_n, stream_, exchange_sync(), wait_kind, signal_kind, routing);
    else if (side == tc::SIDE_NORMS) err = tc::launch_planes<tc::SIDE_NORMS>(problems, n_problems, splits, tile_n, stream_, exchange_sync(), wait_kind, signal_kind, routing);
    else err = tc::launch_planes<tc::SIDE_NONE>(problems, n_problems, splits, tile_n, stream_, exchange_sync(), wait_kind, signal_kind, routing);
    timing_end();
    ++launch_counter_;
    KGE_CUDA(err);
}

// The feature MLP on `n_rows` rows whose hidden buffer holds value + feature . W (src/poplar_kge.cpp:453-458):
// hid = value + relu(concat(value, hid - value) . up) . down, the values read from rows `index[i]` (or
// start + i) of `rows`.  Leaves the MLP's input in `cat` and its pre-activations in `pre` for the backward.
void Engine::launch_mlp_forward(const uint8_t* rows, const uint32_t* index, uint32_t start, unsigned n_rows, int net, float* hid,
                                float* cat, float* pre, float* out) {
    const unsigned D = cfg_.d, M = cfg_.mlp;
    const float* up = dense_ + dense_bounds_[4 + 2 * net];
    const float* down = dense_ + dense_bounds_[5 + 2 * net];
    const dim3 grid(std::min(ceil_div(n_rows * D, 256), 148u * 8));
    if (cfg_.state_type == ST_F32)
        KGE_LAUNCH("mlp", KGE_CUDA(launch_dependent(k_mlp_concat<float>, grid, dim3(256), 0, stream_, rows, layout_, index, start, (int)n_rows, (const float*)hid, cat)));
    else
        KGE_LAUNCH("mlp", KGE_CUDA(launch_dependent(k_mlp_concat<__half>, grid, dim3(256), 0, stream_, rows, layout_, index, start, (int)n_rows, (const float*)hid, cat)));
    SgemmArgs g{};
    g.A = cat; g.lda = 2 * D; g.B = up; g.ldb = M; g.C = pre; g.ldc = M; g.M = (int)n_rows; g.N = (int)M; g.K = (int)(2 * D);
    KGE_LAUNCH("mlp", KGE_CUDA(launch_sgemm(g, stream_)));
    g = SgemmArgs{};
    g.A = pre; g.lda = M; g.a_relu = 1; g.B = down; g.ldb = D; g.C = out; g.ldc = D; g.M = (int)n_rows; g.N = (int)D; g.K = (int)M;
    KGE_LAUNCH("mlp", KGE_CUDA(launch_sgemm(g, stream_)));
    if (cfg_.state_type == ST_F32)
        KGE_LAUNCH("mlp", KGE_CUDA(launch_dependent(k_mlp_finish<float>, grid, dim3(256), 0, stream_, rows, layout_, index, start, (int)n_rows, (const float*)out, hid)));
    else
        KGE_LAUNCH("mlp", KGE_CUDA(launch_dependent(k_mlp_finish<__half>, grid, dim3(256), 0, stream_, rows, layout_, index, start, (int)n_rows, (const float*)out, hid)));
}

// Backward of the MLP for local shard l, after the entity update has left the gradients of the
// MLP's outputs in d_hid_h / d_hid_t and the value's gradient so far in d_val: this shard's
// gradients of the up and down projections go to their owners, the input gradient's first half
// joins d_val, its second half replaces d_hid (the projection gradient's operand), and the rows
// get their Adam step.
void Engine::launch_mlp_backward(unsigned l, unsigned step) {
    ShardBuffers& b = shards_[l];
    const unsigned D = cfg_.d, M = cfg_.mlp, R = cfg_.n_remote();
    const size_t sidx = (size_t)l * cfg_.n_step + step;
    for (unsigned net = 0; net < cfg_.n_net(); ++net) {
        float* d_out = net ? b.d_hid_t : b.d_hid_h;
        const float* up = dense_ + dense_bounds_[4 + 2 * net];
        const float* down = dense_ + dense_bounds_[5 + 2 * net];
        SgemmArgs g{};  // d down = relu(pre)^T . d_out
        g.A = b.mlp_pre[net]; g.lda = M; g.a_trans = 1; g.a_relu = 1; g.B = d_out; g.ldb = D; g.C = b.mlp_dw_down; g.ldc = D;
        g.M = (int)M; g.N = (int)D; g.K = (int)R;
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_sgemm(g, stream_)));
        g = SgemmArgs{};  // d pre = (d_out . down^T) where pre >= 0
        g.A = d_out; g.lda = D; g.B = down; g.ldb = D; g.b_trans = 1; g.C = b.mlp_d_pre; g.ldc = M; g.M = (int)R; g.N = (int)M; g.K = (int)D;
        g.pass = b.mlp_pre[net]; g.ldpass = M;
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_sgemm(g, stream_)));
        g = SgemmArgs{};  // d up = cat^T . d pre
        g.A = b.mlp_cat[net]; g.lda = 2 * D; g.a_trans = 1; g.B = b.mlp_d_pre; g.ldb = M; g.C = b.mlp_dw_up; g.ldc = M;
        g.M = (int)(2 * D); g.N = (int)M; g.K = (int)R;
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_sgemm(g, stream_)));
        g = SgemmArgs{};  // d cat = d pre . up^T
        g.A = b.mlp_d_pre; g.lda = M; g.B = up; g.ldb = M; g.b_trans = 1; g.C = b.mlp_d_cat; g.ldc = 2 * D; g.M = (int)R; g.N = (int)(2 * D); g.K = (int)M;
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_sgemm(g, stream_)));
        const dim3 pgrid(std::min(ceil_div(2 * M * D, 256), 148u * 4));
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_dependent(k_push_dense_rows, pgrid, dim3(256), 0, stream_, (const float*)b.mlp_dw_up, (int)(2 * M),
                                                        (int)(dense_bounds_[4 + 2 * net] / D), (int)D, b.dense_dst, (int)cfg_.world)));
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_dependent(k_push_dense_rows, pgrid, dim3(256), 0, stream_, (const float*)b.mlp_dw_down, (int)M,
                                                        (int)(dense_bounds_[5 + 2 * net] / D), (int)D, b.dense_dst, (int)cfg_.world)));
        const dim3 sgrid(std::min(ceil_div(R * D, 256), 148u * 8));
        KGE_LAUNCH("mlp_bwd", KGE_CUDA(launch_dependent(k_mlp_split, sgrid, dim3(256), 0, stream_, (const float*)b.mlp_d_cat, b.d_val, d_out, (int)R, (int)D)));
    }
    const dim3 agrid(std::min(ceil_div(R * D, 256), 148u * 8));
    const uint8_t* rows_c = b.rows_c2[step & 1];
    const uint32_t* remote = d_remote_ + sidx * R;
    if (cfg_.state_type == ST_F32)
        KGE_LAUNCH("row_adam", KGE_CUDA(launch_dependent(k_row_adam<float>, agrid, dim3(256), 0, stream_, b.table, rows_c, layout_, remote, (const uint32_t*)(d_first_slot_ + sidx * R),
                                                         (const float*)b.d_val, (const float*)(d_step_size_ + step), entity_lr_mod_, adam_, (int)R)));
    else
        KGE_LAUNCH("row_adam", KGE_CUDA(launch_dependent(k_row_adam<__half>, agrid, dim3(256), 0, stream_, b.table, rows_c, layout_, remote, (const uint32_t*)(d_first_slot_ + sidx * R),
                                                         (const float*)b.d_val, (const float*)(d_step_size_ + step), entity_lr_mod_, adam_, (int)R)));
}

// The norm regularisers of local shards' gathered rows (k_regularise): after the hidden rows,
// before the loss (which adds their loss term) and the entity update (which adds their gradients).
void Engine::launch_regularise(unsigned l0, unsigned n, unsigned step) {
    const size_t R = cfg_.n_remote();
    RegParams rp{};
    for (int i = 0; i < 3; ++i) rp.power[i] = cfg_.reg_power[i], rp.weight[i] = cfg_.reg_weight[i];
    rp.loss_scale = cfg_.loss_scale;
    rp.shared = shards_[l0].hid_t == shards_[l0].hid_h ? 1 : 0;
    ShardArgs<RegArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        float* loss = d_reg_loss_ + 2 * (l0 + i);
        shards.s[i] = RegArgs{b.rows_c2[step & 1], b.hid_h, b.hid_t, b.reg_val, b.reg_h, b.reg_t, b.reg_loss_rows, loss, loss + 1, d_reg_counter_ + l0 + i};
    }
    const dim3 grid((unsigned)ceil_div(R, 8), n);
    if (cfg_.state_type == ST_F32) KGE_LAUNCH("regularise", KGE_CUDA(launch_dependent(k_regularise<float>, grid, dim3(256), 0, stream_, shards, layout_, (int)R, rp)));
    else KGE_LAUNCH("regularise", KGE_CUDA(launch_dependent(k_regularise<__half>, grid, dim3(256), 0, stream_, shards, layout_, (int)R, rp)));
}

DropoutParams Engine::dropout_params(unsigned l, unsigned step) const {
    DropoutParams dp{};
    if (!dropout_on()) return dp;
    dp.threshold = (uint32_t)std::lround((1.0 - (double)cfg_.dropout) * 16777216.0);
    dp.seed = cfg_.seed;
    dp.step_key = d_step_key_ + step;
    dp.shard = (uint32_t)(shard0_ + l);
    dp.scale = 1.0f / (1.0f - cfg_.dropout);
    return dp;
}

// hidden = value + dropout(hidden - value) for both calls of local shards (k_dropout_hidden).
void Engine::launch_dropout(unsigned l0, unsigned n, unsigned step) {
    const size_t R = cfg_.n_remote(), quads = ceil_div(cfg_.d, 4);
    ShardArgs<DropoutArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        shards.s[i] = DropoutArgs{b.rows_c2[step & 1], b.hid_h, cfg_.n_net() == 2 ? b.hid_t : b.hid_h, b.hid_t, dropout_params(l0 + i, step)};
    }
    const dim3 grid((unsigned)ceil_div(R * quads, 256), n);
    if (cfg_.state_type == ST_F32) KGE_LAUNCH("dropout", KGE_CUDA(launch_dependent(k_dropout_hidden<float>, grid, dim3(256), 0, stream_, shards, layout_, (int)R)));
    else KGE_LAUNCH("dropout", KGE_CUDA(launch_dependent(k_dropout_hidden<__half>, grid, dim3(256), 0, stream_, shards, layout_, (int)R)));
}

static tc::PlaneOperand plane_operand(const float* hi, const float* lo, long long stride_bytes, bool mn_major) {
    return tc::PlaneOperand{hi, lo, stride_bytes, mn_major ? 1 : 0, 0};
}
// The gathered features of a step as an operand of its contractions.
tc::PlaneOperand Engine::features(const ShardBuffers& b, unsigned step, bool mn_major) const {
    const unsigned parity = step & 1;
    if (cfg_.feature_type == ST_F16) return plane_operand(b.feat_wide2[parity], nullptr, (long long)feat_stride_ * 4, mn_major);
    return plane_operand(reinterpret_cast<const float*>(b.rows_c2[parity] + layout_.off_feat), b.feat_lo2[parity], (long long)layout_.row_bytes, mn_major);
}

// What the lookups of local shard l read: the table's values, or the hidden rows.
LookupRows Engine::lookup_rows(unsigned l, unsigned step) const {
    const ShardBuffers& b = shards_[l];
    const size_t B = cfg_.batch_size, T = cfg_.n_tail(), sidx = (size_t)l * cfg_.n_step + step;
    if (table_lookups_) {
        const uint32_t* row = d_lookup_row_ + sidx * (B + T);
        return LookupRows{b.table, b.table, row, row + B, layout_.row_bytes};
    }
    return LookupRows{reinterpret_cast<const uint8_t*>(b.hid_h), reinterpret_cast<const uint8_t*>(b.hid_t), d_head_ + sidx * B, d_a2a_ + sidx * T, (uint32_t)(cfg_.d * 4)};
}
int Engine::lookup_type() const { return !table_lookups_ ? 0 : cfg_.value_bf16 ? 2 : cfg_.state_type == ST_F16 ? 1 : 0; }

// Lookups, predicted tails and the send half of the exchange for local shards whose hidden rows are ready.
void Engine::launch_lookup(unsigned l0, unsigned n, unsigned step) {
    const bool companion = planes_ && cfg_.dist_fn != DIST_L1 && cfg_.score_fn != SCORE_TRANSH;  // contractions read pred and tails
    const size_t B = cfg_.batch_size, R = cfg_.n_remote();
    LookupSizes sizes{};
    sizes.rel_table = dense_;
    sizes.normal_table = dense_ + dense_bounds_[3];
    sizes.B = (int)B; sizes.T = (int)cfg_.n_tail(); sizes.a2a = (int)cfg_.a2a_size; sizes.D = (int)cfg_.d; sizes.R = (int)R;
    sizes.lo_bf16 = bf16_planes_ ? 1 : 0;
    sizes.prefetch = table_lookups_ && step > 0;  // the first step's index streams come from the kernel in front
    sizes.sync = exchange_sync();
    ShardArgs<LookupArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        const size_t sidx = (size_t)(l0 + i) * cfg_.n_step + step;
        LookupArgs& a = shards.s[i];
        a.rows = lookup_rows(l0 + i, step);
        a.relation = d_relation_ + sidx * B;
        a.send_dst = b.send_dst;
        a.send_lo_dst = companion ? b.send_lo_dst : nullptr;
        a.pred = b.pred;
        a.pred_lo = companion ? b.pred_lo : nullptr;
        a.nrm = b.nrm;
        if (table_lookups_ && (!direct_rows_ || step + 1 == cfg_.n_step)) {  // the regularisers take them, kge_debug_fetch shows the last step's
            a.remote = d_remote_ + sidx * R;
            a.hid = b.hid_h;
        }
    }
    KGE_LAUNCH("lookup", KGE_CUDA(kge::launch_lookup(shards, (int)n, sizes, cfg_.score_fn, lookup_type(), stream_, alone_)));
}

void Engine::launch_lookup_bwd(unsigned l0, unsigned n, unsigned step) {
    const size_t B = cfg_.batch_size;
    ShardArgs<LookupBwdArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        shards.s[i] = LookupBwdArgs{lookup_rows(l0 + i, step), d_relation_ + ((size_t)(l0 + i) * cfg_.n_step + step) * B, b.d_pred, b.d_head, b.d_relrow, b.nrm, b.d_nrm, b.d_normrow};
    }
    KGE_LAUNCH("lookup_bwd", KGE_CUDA(kge::launch_lookup_bwd(shards, (int)n, dense_, dense_ + dense_bounds_[3], (int)B, (int)cfg_.d, cfg_.score_fn, lookup_type(), stream_, alone_)));
}

ShardArgs<TranshScoreArgs> Engine::transh_scores(unsigned l0, unsigned n) const {
    ShardArgs<TranshScoreArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        shards.s[i] = TranshScoreArgs{b.pred, b.nrm, b.tails, b.raw, b.pair_s, b.pair_u};
    }
    return shards;
}
ShardArgs<TranshBwdArgs> Engine::transh_gradients(unsigned l0, unsigned n) const {
    ShardArgs<TranshBwdArgs> shards{};
    for (unsigned i = 0; i < n; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        shards.s[i] = TranshBwdArgs{b.pred, b.nrm, b.tails, b.coeff, b.pair_s, b.pair_u, b.d_pred, b.d_nrm, b.grad_dst,
                                    (int)cfg_.a2a_size, (int)cfg_.batch_size, (int)cfg_.n_tail(), (int)cfg_.d, (int)score_ld_, 0};
    }
    return shards;
}

EntityShard Engine::entity_shard(unsigned l, unsigned step, bool keep_d_hid) const {
    const ShardBuffers& b = shards_[l];
    const size_t B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote(), sidx = (size_t)l * cfg_.n_step + step;
    EntityShard e{};
    e.table = b.table;
    e.rows_c = b.rows_c2[step & 1];
    e.remote = d_remote_ + sidx * R;
    e.perm = d_ent_perm_ + sidx * (B + T);
    e.off = d_ent_off_ + sidx * (R + 1);
    e.first_slot = d_first_slot_ + sidx * R;
    e.d_head = b.d_head;
    e.grad_recv = b.grad_recv;
    if (keep_d_hid) {
        e.d_hid_h = b.d_hid_h;
        e.d_hid_t = b.d_hid_t;
        e.d_hid_h_lo = planes_ ? b.d_hid_h_lo : nullptr;
        e.d_hid_t_lo = planes_ ? b.d_hid_t_lo : nullptr;
    }
    e.heavy = HeavyRows{d_heavy_parts_ + sidx * kHeavySlots, d_heavy_count_ + sidx, b.heavy_partial, b.heavy_counter, d_row_info_ + sidx * 2 * R};
    e.reg_val = b.reg_val;
    e.reg_h = b.reg_h;
    e.reg_t = b.reg_t;
    e.drop = dropout_params(l, step);
    e.defer_grad = b.d_val;
    if (planes_) {
        e.d_relrow[0] = b.d_relrow;
        e.d_relrow[1] = b.d_normrow;
        e.rel_perm = d_rel_perm_ + sidx * B;
        e.rel_off = d_rel_off_ + sidx * (cfg_.n_relation_type + 1);
        e.dense_dst = b.dense_dst;
        e.loss_rows = b.loss_rows;
        e.loss_total = d_loss_total_ + l;
        e.loss_last = d_loss_last_ + l;
        e.extra_loss = d_reg_loss_ ? d_reg_loss_ + 2 * l : nullptr;
    }
    return e;
}
EntityStep Engine::entity_step(unsigned step, unsigned n) const {
    EntityStep g{};
    g.L = layout_;
    g.B = (int)cfg_.batch_size;
    g.R = (int)cfg_.n_remote();
    g.n_shards = (int)n;
    g.step_size = d_step_size_ + step;
    g.lr_modifier = entity_lr_mod_;
    g.ap = adam_;
    g.sync = exchange_sync();
    if (planes_) {
        const int parameter[2] = {0, 3};  // the relation table and TransH's normals
        g.n_rel = (int)cfg_.n_relation_type;
        g.n_tables = cfg_.score_fn == SCORE_TRANSH ? 2 : 1;
        g.n_owner = (int)cfg_.world;
        const unsigned rows = (unsigned)(g.n_rel * g.n_tables);
        g.rel_blocks = (int)(fuse_dense_ ? ceil_div(rows, n) : rows);
        for (int t = 0; t < g.n_tables; ++t) {
            const size_t at = dense_bounds_[parameter[t]];
            g.dense_row0[t] = (int)(at / cfg_.d);
            g.rel_lr_modifier[t] = dense_lr_mod_[parameter[t]];
            if (fuse_dense_) g.rel_w[t] = dense_ + at, g.rel_m[t] = dense_m_ + at, g.rel_v[t] = dense_v_ + at;
        }
    }
    return g;
}

// The training step of batched launches: five to nine on the step's chain (hidden rows, lookups + send, scores, loss, score
// gradients + return, the prediction's backward, segment sums + Adam + relation gradients, projection gradient, dense
// update; what a model has no use for is left out, and the lookups of the elementwise score functions are the hidden
// kernel's epilogue) and the next step's gather beside the last two.  Every launch works on all local shards, which meet
// at the exchange (the tails and the tails' gradients), and every operand of a contraction is the fp32 array its producer
// wrote (the upper TF32 plane) plus a lower plane the same producer wrote next to it.
// With a stream per shard instead, forked and joined three times a step, and a dense update of its own (us per step,
// before -> after): demo preset, 2 shards, 40.4 -> 32.3; four shards of 256 x 320 L1 scores, 70.0 -> 67.2; four of 256 x 512
// fp16 rows, 79.4 -> 83.1 (57.4 with the pair gradients of today); two shards of the headline step 129.5 -> 112.9.
void Engine::launch_step_planes(unsigned step, const LossParams& lp, float normaliser) {
    const unsigned B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote(), D = cfg_.d, F = cfg_.f;
    const unsigned n_rel = cfg_.n_relation_type, parity = step & 1, n_nets = cfg_.n_net(), ld = score_ld_;
    const bool transh = cfg_.score_fn == SCORE_TRANSH, dot = cfg_.dist_fn == DIST_DOT && !transh, l2 = cfg_.dist_fn == DIST_L2 && !transh;
    // bf16 embeddings: the dot-product scores and their gradients multiply bfloat16 copies of pred,
    // tails and the coefficients (written by their producers into the companion planes)
    const bool bf16 = bf16_planes_;
    auto plane16 = [](const float* values, long long row_elems, bool mn_major) {
        return tc::PlaneOperand{values, nullptr, row_elems * 2, mn_major ? 1 : 0, 2};
    };
    const ExchangeSync sync = exchange_sync();
    auto step_ptr = [&](uint32_t* base, unsigned l, size_t per_step) { return base + ((size_t)l * cfg_.n_step + step) * per_step; };
    tc::PlaneProblem problems[tc::kMaxPlaneProblems];

    // 1. hidden = value + feature . W, and (elementwise score functions) from its epilogue the lookups and the send half of the exchange
    const bool fused_route = F > 0 && (cfg_.score_fn == SCORE_TRANSE || cfg_.score_fn == SCORE_DISTMULT) && !dropout_on();
    // rows with many lookups are routed in parts by a kernel of their own, which then publishes the tails
    const bool heavy_route = fused_route && split_popular_rows_ && heavy_route_;
    shards_fork();
    for (unsigned l0 = 0; l0 < n_local_; l0 += group_) {
        const ShardScope on_stream(*this, l0 / group_);
        const unsigned n = std::min(group_, n_local_ - l0);
        if (F > 0) {
            tc::RouteArgs routes[kShardBatch] = {};
            for (unsigned i = 0; i < n; ++i) {
                const ShardBuffers& b = shards_[l0 + i];
                const size_t sidx = (size_t)(l0 + i) * cfg_.n_step + step;
                for (unsigned net = 0; net < n_nets; ++net) {
                    tc::PlaneProblem& p = problems[i * n_nets + net];
                    p = tc::PlaneProblem{};
                    const size_t w = dense_bounds_[1 + net];
                    p.A = features(b, step, false);
                    p.B = plane_operand(dense_ + w, dense_lo_ + w, (long long)D * 4, true);
                    tc::GemmArgs& g = p.g;
                    g.M = (int)R; g.N = (int)D; g.K = (int)F;
                    g.epilogue = tc::EPI_ADD_TABLE_VALUE;
                    g.out = net ? b.hid_t : b.hid_h; g.ldc = D; g.block_rows = 1;
                    g.x_base = b.rows_c2[parity]; g.x_row_stride_bytes = layout_.row_bytes;
                    g.x_is_half = cfg_.value_bf16 ? 2 : (cfg_.state_type == ST_F16 ? 1 : 0);
                }
                tc::RouteArgs& route = routes[i];
                route.perm = d_ent_perm_ + sidx * (B + T);
                route.off = d_ent_off_ + sidx * (R + 1);
                route.relation = step_ptr(d_relation_, l0 + i, B);
                route.rel_table = dense_;
                route.send_dst = b.send_dst;
                route.send_lo_dst = b.send_lo_dst;
                route.pred = b.pred;
                route.pred_lo = b.pred_lo;
                route.B = (int)B; route.a2a = (int)cfg_.a2a_size; route.n_shard = (int)cfg_.n_shard; route.score_fn = cfg_.score_fn;
                route.lo_bf16 = bf16 ? 1 : 0;
                route.first_slot = heavy_route ? step_ptr(d_first_slot_, l0 + i, R) : nullptr;
            }
            const tc::Routing routing{routes, (int)n, (int)n_nets, {n_nets == 2 ? 1 : 3, 2}};
            launch_planes("hidden", problems, (int)(n * n_nets), tc::SIDE_NONE, XCHG_DENSE_PARAMS, fused_route && !heavy_route ? XCHG_TAILS : -1,
                          fused_route ? &routing : nullptr);
        } else {
            launch_exchange_wait(XCHG_DENSE_PARAMS);
        }
        if (heavy_route)
            for (unsigned l = l0; l < l0 + n; ++l) {
                const ShardBuffers& b = shards_[l];
                const size_t sidx = (size_t)l * cfg_.n_step + step;
                KGE_LAUNCH("route_heavy", KGE_CUDA(launch_dependent(k_route_heavy, dim3(kHeavySlots), dim3(256), 0, stream_, (const float*)b.hid_h, (const float*)b.hid_t,
                                                                    (const uint4*)(d_heavy_parts_ + sidx * kHeavySlots), (const uint32_t*)(d_heavy_count_ + sidx),
                                                                    (const uint32_t*)(d_ent_perm_ + sidx * (B + T)), (const uint32_t*)step_ptr(d_relation_, l, B),
                                                                    (const float*)dense_, b.send_dst, b.send_lo_dst, b.pred, b.pred_lo, (int)B, (int)cfg_.a2a_size,
                                                                    (int)D, cfg_.score_fn, bf16 ? 1 : 0, sync)));
            }
        if (dropout_on()) launch_dropout(l0, n, step);
        if (!fused_route) launch_lookup(l0, n, step);
        if (cfg_.regularised()) launch_regularise(l0, n, step);
    }
    shards_join();
    KGE_CUDA(cudaGetLastError());

    shards_fork();
    for (unsigned l0 = 0; l0 < n_local_; l0 += group_) {
        const ShardScope on_stream(*this, l0 / group_);
        const unsigned n = std::min(group_, n_local_ - l0);
        // 2. scores
        if (transh) {
            KGE_LAUNCH("score", KGE_CUDA(launch_transh_score(transh_scores(l0, n), (int)n, (int)B, (int)T, (int)D, (int)ld, sync, stream_)));
        } else if (dot || (l2 && cfg_.l2_contraction)) {
            // (the L2 distance as |p|^2 + |t|^2 - 2 p.t, in the direct form where that cancels)
            for (unsigned i = 0; i < n; ++i) {
                const ShardBuffers& b = shards_[l0 + i];
                tc::PlaneProblem& p = problems[i];
                p = tc::PlaneProblem{};
                p.A = bf16 ? plane16(b.pred_lo, D, false) : plane_operand(b.pred, b.pred_lo, (long long)D * 4, false);
                p.B = bf16 ? plane16(b.tails_lo, D, false) : plane_operand(b.tails, b.tails_lo, (long long)D * 4, false);
                p.g.M = (int)B; p.g.N = (int)T; p.g.K = (int)D;
                p.g.epilogue = dot ? tc::EPI_STORE : tc::EPI_L2_DISTANCE;
                p.g.out = b.raw; p.g.ldc = ld; p.g.block_rows = 1;
            }
            launch_planes("score", problems, (int)n, dot ? tc::SIDE_NONE : tc::SIDE_NORMS, XCHG_TAILS, -1);
        } else {
            ShardArgs<ScoreArgs> shards{};
            for (unsigned i = 0; i < n; ++i) shards.s[i] = ScoreArgs{shards_[l0 + i].pred, shards_[l0 + i].tails, shards_[l0 + i].raw};
            KGE_LAUNCH("score", KGE_CUDA(launch_score(cfg_.dist_fn, shards, (int)n, (int)B, (int)T, (int)D, (int)ld, stream_, sync)));
        }
        // 3. loss and the coefficients of the score gradients (the rows' loss terms are added up by a block of the entity update, off the chain)
        ShardArgs<LossArgs> loss{};
        for (unsigned i = 0; i < n; ++i) {
            const ShardBuffers& b = shards_[l0 + i];
            loss.s[i] = LossArgs{b.raw, step_ptr(d_tail_, l0 + i, B), b.coeff, dot || l2 ? b.coeff_lo : nullptr, b.loss_rows, nullptr, nullptr, nullptr, nullptr};
        }
        KGE_LAUNCH("loss", KGE_CUDA(launch_loss(loss, (int)n, lp, 1.0f / normaliser, bf16 ? 1 : 0, (int)B, stream_, alone_)));
        // 4. score gradients; the tails' rows go straight to the shards that own them
        if (transh) {
            KGE_LAUNCH("score_bwd", KGE_CUDA(launch_transh_bwd(transh_gradients(l0, n), (int)n, stream_)));
            launch_exchange_signal(XCHG_TAIL_GRADS);
        } else if (!dot && !l2) {
            ShardArgs<PairBwdArgs> shards{};
            for (unsigned i = 0; i < n; ++i) {
                const ShardBuffers& b = shards_[l0 + i];
                PairBwdArgs& pa = shards.s[i];
                pa.D = (int)D;
                pa.p[0] = {b.pred, b.tails, b.coeff, (int)B, (int)T, (int)ld, 1, b.d_pred, nullptr, 1};
                pa.p[1] = {b.tails, b.pred, b.coeff, (int)T, (int)B, 1, (int)ld, nullptr, b.grad_dst, (int)cfg_.a2a_size};
            }
            KGE_LAUNCH("score_bwd", KGE_CUDA(launch_pair_bwd(DIST_L1, shards, (int)n, stream_)));
            launch_exchange_signal(XCHG_TAIL_GRADS);
        } else {
            //   dot:  d_pred = C . tails,                          d_tails = C^T . pred
            //   L2:   d_pred = rowsum(C) * pred - C . tails,       d_tails = colsum(C) * tails - C^T . pred
            for (unsigned i = 0; i < n; ++i) {
                const ShardBuffers& b = shards_[l0 + i];
                tc::PlaneProblem &g = problems[2 * i], &h = problems[2 * i + 1];
                g = h = tc::PlaneProblem{};
                g.A = bf16 ? plane16(b.coeff_lo, ld, false) : plane_operand(b.coeff, b.coeff_lo, (long long)ld * 4, false);
                g.B = bf16 ? plane16(b.tails_lo, D, true) : plane_operand(b.tails, b.tails_lo, (long long)D * 4, true);
                g.g.M = (int)B; g.g.N = (int)D; g.g.K = (int)T;
                g.g.epilogue = l2 ? tc::EPI_ROWSUM_X_MINUS : tc::EPI_STORE;
                g.g.out = b.d_pred; g.g.ldc = D; g.g.block_rows = 1;
                g.g.x_base = reinterpret_cast<const uint8_t*>(b.pred); g.g.x_row_stride_bytes = (long long)D * 4;
                h.A = bf16 ? plane16(b.coeff_lo, ld, true) : plane_operand(b.coeff, b.coeff_lo, (long long)ld * 4, true);
                h.B = bf16 ? plane16(b.pred_lo, D, true) : plane_operand(b.pred, b.pred_lo, (long long)D * 4, true);
                h.g.M = (int)T; h.g.N = (int)D; h.g.K = (int)B;
                h.g.epilogue = g.g.epilogue;
                h.g.out = nullptr; h.g.out_blocks = b.grad_dst; h.g.block_rows = (int)cfg_.a2a_size; h.g.ldc = D;
                h.g.x_base = reinterpret_cast<const uint8_t*>(b.tails); h.g.x_row_stride_bytes = (long long)D * 4;
            }
            launch_planes("score_bwd", problems, (int)(2 * n), l2 ? tc::SIDE_ROWSUM : tc::SIDE_NONE, -1, XCHG_TAIL_GRADS);
        }
        if (cfg_.score_fn != SCORE_TRANSE) launch_lookup_bwd(l0, n, step);
    }
    shards_join();
    KGE_CUDA(cudaGetLastError());

    // 5. segment sums + row-wise Adam, and the relation rows of the dense gradient
    const bool gather_ahead = step + 1 < cfg_.n_step && !direct_rows_;
    const bool gather_beside = gather_ahead && (side_streams_ & 2u);
    // with the table's own rows nothing reads the hidden rows' gradients but kge_debug_fetch, which shows the last step's
    const bool keep_d_hid = !direct_rows_ || step + 1 == cfg_.n_step;
    const bool extras = cfg_.regularised() || dropout_on();
    shards_fork();
    for (unsigned l0 = 0; l0 < n_local_; l0 += group_) {
        const ShardScope on_stream(*this, l0 / group_);
        const unsigned n = std::min(group_, n_local_ - l0);
        ShardArgs<EntityShard> shards{};
        for (unsigned i = 0; i < n; ++i) shards.s[i] = entity_shard(l0 + i, step, keep_d_hid);
        EntityStep es = entity_step(step, n);
        es.inv_normaliser = 1.0f / normaliser;
        auto update = [&](auto state) {
            using ST = decltype(state);
            if (extras) return launch_entity_update<ST, 4, true>(shards, es, stream_);
            if (direct_rows_) return launch_entity_update<ST, 4, false, true>(shards, es, stream_);
            return launch_entity_update<ST, 4>(shards, es, stream_);
        };
        KGE_LAUNCH("entity_update", KGE_CUDA(cfg_.state_type == ST_F32 ? update(float{}) : update(__half{})));
        if (gather_beside) launch_gather(step + 1, l0, n, side_begin());
    }
    KGE_CUDA(cudaGetLastError());
    if (gather_beside) side_end(1);
    // 6. d W = feature^T . d_hidden: the projection's Adam step, over the rows of all shards, or straight into the owners'
    // slices of each shard's partial dense gradient
    const unsigned at_once = fuse_dense_ ? n_local_ : group_;
    for (unsigned l0 = 0; l0 < n_local_; l0 += at_once) {
        const ShardScope on_stream(*this, l0 / group_);
        const unsigned n = std::min(at_once, n_local_ - l0);
        if (F > 0) launch_projection_bwd(l0, n, step, fuse_dense_);
        else launch_exchange_signal(XCHG_DENSE_PARTIALS);  // the relation rows of the entity update are all there is
    }
    shards_join();
    KGE_CUDA(cudaGetLastError());
    if (gather_ahead && !gather_beside) launch_gather(step + 1, stream_);
    // 7. dense parameters: reduce over shards, Adam on the owned rows, new values and their lower planes into every replica
    if (!fuse_dense_) launch_dense_update(step);
    KGE_CUDA(cudaGetLastError());
    if (gather_beside) side_join(1);
}

// d W = feature^T . d_hidden of local shards l0 .. l0 + n - 1.  `update`: one contraction over the rows of all of them (shard
// behind shard in memory), which ends in the projection's Adam step; else each shard's goes to the owners' slices of its
// partial dense gradient.
void Engine::launch_projection_bwd(unsigned l0, unsigned n, unsigned step, bool update) {
    const unsigned R = cfg_.n_remote(), D = cfg_.d, F = cfg_.f, n_nets = cfg_.n_net(), n_problems = update ? 1 : n;
    tc::PlaneProblem problems[tc::kMaxPlaneProblems];
    for (unsigned i = 0; i < n_problems; ++i) {
        const ShardBuffers& b = shards_[l0 + i];
        for (unsigned net = 0; net < n_nets; ++net) {
            tc::PlaneProblem& p = problems[i * n_nets + net];
            p = tc::PlaneProblem{};
            p.A = features(b, step, true);
            p.B = plane_operand(net ? b.d_hid_t : b.d_hid_h, net ? b.d_hid_t_lo : b.d_hid_h_lo, (long long)D * 4, true);
            tc::GemmArgs& g = p.g;
            g.M = (int)F; g.N = (int)D; g.K = (int)(update ? n * R : R);
            g.block_row_offset = (int)(cfg_.n_relation_type + net * F); g.block_rows = 1; g.ldc = D;
            if (update) {
                g.epilogue = tc::EPI_DENSE_ADAM;
                g.x_base = reinterpret_cast<const uint8_t*>(dense_ + dense_bounds_[1 + net]);
                g.x_row_stride_bytes = (long long)D * 4;
                g.adam = tc::DenseAdamArgs{dense_, dense_lo_, dense_m_, dense_v_, d_step_size_ + step, dense_lr_mod_[1 + net], adam_.beta_m, adam_.beta_v,
                                           adam_.one_minus_beta_m, adam_.one_minus_beta_v, adam_.epsilon, adam_.weight_decay};
            } else {
                g.epilogue = tc::EPI_STORE;
                g.out_blocks = b.dense_dst; g.block_cyclic = (int)cfg_.world;
            }
        }
    }
    launch_planes("projection_bwd", problems, (int)(n_problems * n_nets), tc::SIDE_NONE, -1, XCHG_DENSE_PARTIALS);
}

// Where the dense Adam steps are taken by the kernels that produce the gradients, these are never stored: the last step's
// partial dense gradient of local shard l, from what that step has left of its operands (kge_debug_fetch).
void Engine::restore_dense_partial(unsigned l) {
    if (!staged_ || stage_fresh_)
        fail(KGE_INVALID_ARGUMENT, "kge_debug_fetch: 'dense_grad' is made from the index streams of the last run: there has been none, or a newly staged batch has replaced them");
    ShardBuffers& b = shards_[l];
    const unsigned step = cfg_.n_step - 1, n_rel = cfg_.n_relation_type;
    const size_t sidx = (size_t)l * cfg_.n_step + step;
    const float* per_triple[2] = {b.d_relrow, b.d_normrow};
    struct Untimed {  // (these launches belong to no run)
        bool &timing, before;
        ~Untimed() { timing = before; }
    } untimed{kernel_timing_, std::exchange(kernel_timing_, false)};
    for (int table = 0; table < (cfg_.score_fn == SCORE_TRANSH ? 2 : 1); ++table)
        KGE_CUDA(launch_dependent(k_dense_partial<4>, dim3(n_rel), dim3(64 * kRelationLanes), 0, stream_, per_triple[table], d_rel_perm_ + sidx * cfg_.batch_size,
                                  d_rel_off_ + sidx * (n_rel + 1), (int)n_rel, (int)cfg_.d, b.proj_partial, 0, 1, proj_elems_, b.dense_dst, (int)cfg_.world,
                                  exchange_sync(), -1, table ? (int)(dense_bounds_[3] / cfg_.d) : 0));
    if (cfg_.f) launch_projection_bwd(l, 1, step, false);
}

// Dense parameters: every process, also one that owns nothing, launches it, since the kernel carries two hand-overs.
void Engine::launch_dense_update(unsigned step) {
    DenseUpdateArgs da{};
    da.sync = exchange_sync();
    da.partials = d_partials_;
    da.n_partial = (int)cfg_.n_shard;
    da.replicas = d_replicas_;
    da.replicas_lo = planes_ ? d_replicas_lo_ : nullptr;
    da.n_replica = (int)cfg_.world;
    da.adam_m = dense_m_;
    da.adam_v = dense_v_;
    da.n_own = own_rows_;
    da.row_width = cfg_.d;
    for (int i = 0; i <= kDenseParams; ++i) da.bounds[i] = dense_bounds_[i];
    for (int i = 0; i < kDenseParams; ++i) da.lr_modifier[i] = dense_lr_mod_[i];
    da.step_size = d_step_size_ + step;
    da.ap = adam_;
    // The parameter itself is read from this process's own replica (entry `rank`).
    const unsigned blocks = (unsigned)std::min<size_t>((own_rows_ * cfg_.d / (cfg_.d % 4 == 0 ? 4 : 1) + 255) / 256, 148 * 8);
    KGE_LAUNCH("dense_update", KGE_CUDA(launch_dependent(k_dense_update, dim3(std::max(1u, blocks)), dim3(256), 0, stream_, da, (int)cfg_.rank)));
}

void Engine::launch_one_step(unsigned step) {
    const unsigned B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote(), D = cfg_.d, F = cfg_.f;
    const unsigned n_rel = cfg_.n_relation_type;
    const bool two_nets = cfg_.n_net() == 2;
    const bool vec = (D % 4) == 0;
    const float* W0 = cfg_.n_net() >= 1 ? dense_ + dense_bounds_[1] : nullptr;
    const float* W1 = two_nets ? dense_ + dense_bounds_[2] : W0;
    const bool transh = cfg_.score_fn == SCORE_TRANSH;

    LossParams lp{};
    lp.loss_fn = cfg_.loss_fn;
    lp.score_fn = cfg_.score_fn;
    lp.dist_fn = cfg_.dist_fn;
    lp.n_tail = (int)T;
    lp.ld = (int)score_ld_;
    lp.gamma = cfg_.gamma;
    lp.adversarial_scale = cfg_.adversarial_scale;
    lp.w_neg = (0.5f * (float)T) / (float)(T - 1);
    lp.w_pos = 0.5f * (float)T;
    float normaliser;
    if (cfg_.loss_fn == LOSS_LOGSIGMOID) {
        normaliser = (float)(cfg_.n_shard * B * cfg_.a2a_size * cfg_.n_shard);
        lp.softmax_shift = 0.f;
    } else {
        normaliser = (float)(cfg_.n_shard * B);
        const float correction = (float)(std::log((double)(cfg_.n_entity * cfg_.n_shard - 1)) -
                                         std::log((double)(cfg_.n_shard * cfg_.a2a_size - 1)));
        lp.softmax_shift = cfg_.correction_weight != 0.f ? cfg_.correction_weight * correction : 0.f;
    }
    lp.grad_scale = cfg_.loss_scale / normaliser;

    if (planes_) return launch_step_planes(step, lp, normaliser);
    const ExchangeSync sync = exchange_sync();
    const bool proj_direct = cfg_.tensor_cores && F > 0;  // the projection gradient lands in the partial dense vector directly
    auto step_ptr = [&](uint32_t* base, unsigned l, size_t per_step) {
        return base + ((size_t)l * cfg_.n_step + step) * per_step;
    };

    // 1./2. hidden rows, lookups, send half of the exchange
    shards_fork();
    for (unsigned l = 0; l < n_local_; ++l) {
        const ShardScope on_stream(*this, l);
        ShardBuffers& b = shards_[l];
        uint8_t* rows_c = b.rows_c2[step & 1];
        if (cfg_.tensor_cores && F > 0) {
            // hidden = value + feature . W on the tensor cores: A = gathered feature rows, B = W stored [F, D]
            tc::GemmArgs nets[2] = {};
            const int n_nets = two_nets ? 2 : 1;
            for (int net = 0; net < n_nets; ++net) {
                tc::GemmArgs& g = nets[net];
                g.A = tc::make_operand(rows_c + layout_.off_feat, layout_.row_bytes, cfg_.feature_type == ST_F16, false);
                g.B = tc::make_operand(net ? W1 : W0, (long long)D * 4, false, true);
                g.M = (int)R; g.N = (int)D; g.K = (int)F; g.k_per_split = (int)round_up(F, 32);
                g.epilogue = tc::EPI_ADD_TABLE_VALUE;
                g.out = net ? b.hid_t : b.hid_h; g.ldc = D; g.block_rows = 1;
                g.x_base = rows_c; g.x_row_stride_bytes = layout_.row_bytes; g.x_gather = nullptr;
                g.x_is_half = cfg_.value_bf16 ? 2 : (cfg_.state_type == ST_F16 ? 1 : 0);
            }
            // the projection was updated by the processes that own its slices
            launch_tc("hidden", nets, n_nets, tc_splits(n_nets * ceil_div(R, 128) * ceil_div(D, 64), F), cfg_.feature_type == ST_F16, false,
                      XCHG_DENSE_PARAMS, -1);
        } else {
            launch_exchange_wait(XCHG_DENSE_PARAMS);
            dim3 grid(ceil_div(R, 64), ceil_div(D, 64), two_nets ? 2 : 1);
            KGE_LAUNCH("hidden", KGE_DISPATCH_ROW(cfg_, KGE_CUDA(launch_dependent(k_hidden<ST, FT>, dim3(grid), dim3(256), 0, stream_, 
                                                            rows_c, layout_, nullptr, 0u, (int)R, W0, W1, b.hid_h, b.hid_t))));
        }
        if (mlp_on())
            for (unsigned net = 0; net < cfg_.n_net(); ++net)
                launch_mlp_forward(rows_c, nullptr, 0u, R, (int)net, net ? b.hid_t : b.hid_h, b.mlp_cat[net], b.mlp_pre[net], b.mlp_out);
        if (dropout_on()) launch_dropout(l, 1, step);
        launch_lookup(l, 1, step);
        if (cfg_.regularised()) launch_regularise(l, 1, step);
    }
    shards_join();
    KGE_CUDA(cudaGetLastError());

    // 3./4./5a. scores, loss, score backward with the return half of the exchange
    shards_fork();
    for (unsigned l = 0; l < n_local_; ++l) {
        const ShardScope on_stream(*this, l);
        ShardBuffers& b = shards_[l];
        const uint32_t* tail = step_ptr(d_tail_, l, B);
        PairBwdArgs pa{};
        pa.D = (int)D;
        pa.p[0] = {b.pred, b.tails, b.coeff, (int)B, (int)T, (int)T, 1, b.d_pred, nullptr, 1};
        pa.p[1] = {b.tails, b.pred, b.coeff, (int)T, (int)B, 1, (int)T, nullptr, b.grad_dst, (int)cfg_.a2a_size};
        const bool tc_score = cfg_.tensor_cores && cfg_.dist_fn == DIST_DOT;
        const bool tc_bwd = cfg_.tensor_cores && cfg_.dist_fn != DIST_L1;
        if (transh) {
            KGE_LAUNCH("score", KGE_CUDA(launch_transh_score(transh_scores(l, 1), 1, (int)B, (int)T, (int)D, (int)score_ld_, sync, stream_)));
        } else if (tc_score) {
            tc::GemmArgs g{};
            g.A = tc::make_operand(b.pred, (long long)D * 4, false, false);
            g.B = tc::make_operand(b.tails, (long long)D * 4, false, false);
            g.M = (int)B; g.N = (int)T; g.K = (int)D; g.k_per_split = (int)round_up(D, 32);
            g.epilogue = tc::EPI_STORE; g.out = b.raw; g.ldc = T; g.block_rows = 1;
            launch_tc("score", &g, 1, tc_splits(ceil_div(B, 128) * ceil_div(T, 64), D), false, false, XCHG_TAILS, -1);
        } else {
            // the tail rows come from the other processes: the 16-byte-copy kernel waits for them itself
            const bool fused_wait = score_rows_aligned(b.pred, b.tails, (int)D);
            if (!fused_wait) launch_exchange_wait(XCHG_TAILS);
            KGE_LAUNCH("score", KGE_CUDA(launch_score(cfg_.dist_fn, b.pred, b.tails, b.raw, (int)B, (int)T, (int)D, stream_,
                                                      fused_wait ? sync : ExchangeSync{})));
        }
        ShardArgs<LossArgs> loss{};
        loss.s[0] = LossArgs{b.raw, tail, b.coeff, nullptr, b.loss_rows, d_loss_total_ + l, d_loss_last_ + l, d_loss_counter_ + l, d_reg_loss_ ? d_reg_loss_ + 2 * l : nullptr};
        KGE_LAUNCH("loss", KGE_CUDA(launch_loss(loss, 1, lp, 1.0f / normaliser, 0, (int)B, stream_, alone_ && transh)));
        if (tc_bwd) {
            // Both input gradients are contractions with the coefficient matrix C [B, T]:
            //   dot:  d_pred = C . tails,                          d_tails = C^T . pred
            //   L2:   d_pred = rowsum(C) * pred - C . tails,       d_tails = colsum(C) * tails - C^T . pred
            // (sum_j C_ij (p_i - t_j) written out; C already holds gradient / distance).
            const bool l2 = cfg_.dist_fn == DIST_L2;
            tc::GemmArgs both[2] = {};
            tc::GemmArgs& g = both[0];
            g.A = tc::make_operand(b.coeff, (long long)T * 4, false, false);
            g.B = tc::make_operand(b.tails, (long long)D * 4, false, true);
            g.M = (int)B; g.N = (int)D; g.K = (int)T; g.k_per_split = (int)round_up(T, 32);
            g.epilogue = l2 ? tc::EPI_ROWSUM_X_MINUS : tc::EPI_STORE;
            g.out = b.d_pred; g.ldc = D; g.block_rows = 1;
            g.x_base = reinterpret_cast<const uint8_t*>(b.pred); g.x_row_stride_bytes = (long long)D * 4;
            tc::GemmArgs& h = both[1];
            h.A = tc::make_operand(b.coeff, (long long)T * 4, false, true);
            h.B = tc::make_operand(b.pred, (long long)D * 4, false, true);
            h.M = (int)T; h.N = (int)D; h.K = (int)B; h.k_per_split = (int)round_up(std::max(B, T), 32);
            h.epilogue = l2 ? tc::EPI_ROWSUM_X_MINUS : tc::EPI_STORE;
            h.out = nullptr; h.out_blocks = b.grad_dst; h.block_rows = (int)cfg_.a2a_size; h.ldc = D;
            h.x_base = reinterpret_cast<const uint8_t*>(b.tails); h.x_row_stride_bytes = (long long)D * 4;
            g.k_per_split = h.k_per_split;
            launch_tc("score_bwd", both, 2, tc_splits((ceil_div(B, 128) + ceil_div(T, 128)) * ceil_div(D, 64), std::min(B, T)), false, l2,
                      -1, XCHG_TAIL_GRADS);
        } else if (transh) {
            KGE_LAUNCH("score_bwd", KGE_CUDA(launch_transh_bwd(transh_gradients(l, 1), 1, stream_)));
            launch_exchange_signal(XCHG_TAIL_GRADS);
        } else {
            KGE_LAUNCH("score_bwd", KGE_CUDA(launch_pair_bwd(cfg_.dist_fn, pa, stream_)));
            launch_exchange_signal(XCHG_TAIL_GRADS);
        }
        if (cfg_.score_fn != SCORE_TRANSE) launch_lookup_bwd(l, 1, step);
        if (transh) {
            // the normals' rows of the partial dense gradient, behind the relation table and the projections
            const size_t sidx = (size_t)l * cfg_.n_step + step;
            const int normal_row0 = (int)(n_rel + cfg_.n_net() * F);
            if (vec)
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<4>, dim3(n_rel), dim3(64 * kRelationLanes), 0, stream_,
                                                b.d_normrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, 0, 1, proj_elems_, b.dense_dst, (int)cfg_.world, sync, -1, normal_row0)));
            else
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<1>, dim3(n_rel), dim3(64 * kRelationLanes), 0, stream_,
                                                b.d_normrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, 0, 1, proj_elems_, b.dense_dst, (int)cfg_.world, sync, -1, normal_row0)));
        }
    }
    shards_join();
    KGE_CUDA(cudaGetLastError());

    if (proj_direct) {
        // The relation gradients depend on the score backward only: they are summed beside the entity update.
        const unsigned saved = side_streams_;
        side_streams_ = saved & 1u;
        cudaStream_t side = side_begin();
        for (unsigned l = 0; l < n_local_; ++l) {
            ShardBuffers& b = shards_[l];
            const size_t sidx = (size_t)l * cfg_.n_step + step;
            if (vec)
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<4>, dim3(n_rel), dim3(64 * kRelationLanes), 0, side,
                                                b.d_relrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, 0, 1, proj_elems_, b.dense_dst, (int)cfg_.world, sync, -1, 0)));
            else
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<1>, dim3(n_rel), dim3(64 * kRelationLanes), 0, side,
                                                b.d_relrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, 0, 1, proj_elems_, b.dense_dst, (int)cfg_.world, sync, -1, 0)));
        }
        side_end(0);
        side_streams_ = saved;
    }

    // 5b. segment sums + row-wise Adam; projection and relation gradients of this shard
    const bool gather_ahead = step + 1 < cfg_.n_step;
    const bool gather_beside = gather_ahead && (side_streams_ & 2u);
    shards_fork();
    for (unsigned l = 0; l < n_local_; ++l) {
        const ShardScope on_stream(*this, l);
        ShardBuffers& b = shards_[l];
        ShardArgs<EntityShard> shard{};
        shard.s[0] = entity_shard(l, step, true);
        const EntityStep es = entity_step(step, 1);
        const bool extras = cfg_.regularised() || dropout_on() || mlp_on();
        if (cfg_.state_type == ST_F32) {
            if (vec) KGE_LAUNCH("entity_update", KGE_CUDA((extras ? launch_entity_update<float, 4, true>(shard, es, stream_) : launch_entity_update<float, 4>(shard, es, stream_))));
            else KGE_LAUNCH("entity_update", KGE_CUDA((extras ? launch_entity_update<float, 1, true>(shard, es, stream_) : launch_entity_update<float, 1>(shard, es, stream_))));
        } else {
            if (vec) KGE_LAUNCH("entity_update", KGE_CUDA((extras ? launch_entity_update<__half, 4, true>(shard, es, stream_) : launch_entity_update<__half, 4>(shard, es, stream_))));
            else KGE_LAUNCH("entity_update", KGE_CUDA((extras ? launch_entity_update<__half, 1, true>(shard, es, stream_) : launch_entity_update<__half, 1>(shard, es, stream_))));
        }
        if (mlp_on()) launch_mlp_backward(l, step);
        // the next step's rows: needs only the rows just updated, runs beside the rest of this step
        if (gather_beside) launch_gather(step + 1, l, 1, side_begin());
    }
    KGE_CUDA(cudaGetLastError());
    if (gather_beside) side_end(1);
    for (unsigned l = 0; l < n_local_; ++l) {
        const ShardScope on_stream(*this, l);
        ShardBuffers& b = shards_[l];
        uint8_t* rows_c = b.rows_c2[step & 1];
        const size_t sidx = (size_t)l * cfg_.n_step + step;
        if (F > 0 && cfg_.tensor_cores) {
            // d W = feature^T . d_hidden: the gathered rows are the k index of both operands
            tc::GemmArgs nets[2] = {};
            for (unsigned net = 0; net < cfg_.n_net(); ++net) {
                tc::GemmArgs& g = nets[net];
                g.A = tc::make_operand(rows_c + layout_.off_feat, layout_.row_bytes, cfg_.feature_type == ST_F16, true);
                g.B = tc::make_operand(net ? b.d_hid_t : b.d_hid_h, (long long)D * 4, false, true);
                g.M = (int)F; g.N = (int)D; g.K = (int)R; g.k_per_split = proj_rows_per_split_;
                g.epilogue = tc::EPI_STORE;
                // straight into this shard's partial dense gradient, behind the relation rows: row m of
                // the projection is row n_rel + net * F + m of the dense vector, and goes to its owner
                g.out = nullptr; g.out_blocks = b.dense_dst; g.block_rows = 1; g.block_cyclic = (int)cfg_.world;
                g.block_row_offset = (int)(n_rel + net * F); g.ldc = D;
            }
            launch_tc("projection_bwd", nets, (int)cfg_.n_net(),
                      tc_splits(cfg_.n_net() * ceil_div(F, 128) * ceil_div(D, 64), R), cfg_.feature_type == ST_F16, false,
                      -1, XCHG_DENSE_PARTIALS);
        } else if (F > 0) {
            dim3 grid(ceil_div(F, 64), ceil_div(D, 64), cfg_.n_net() * proj_splits_);
            const float* dh1 = two_nets ? b.d_hid_t : b.d_hid_h;
            if (cfg_.feature_type == ST_F32)
                KGE_LAUNCH("projection_bwd", KGE_CUDA(launch_dependent(k_projection_bwd<float>, dim3(grid), dim3(256), 0, stream_, 
                                                 rows_c, layout_, nullptr, (int)R, b.d_hid_h, dh1, proj_splits_,
                                                 proj_rows_per_split_, b.proj_partial)));
            else
                KGE_LAUNCH("projection_bwd", KGE_CUDA(launch_dependent(k_projection_bwd<__half>, dim3(grid), dim3(256), 0, stream_, 
                                                 rows_c, layout_, nullptr, (int)R, b.d_hid_h, dh1, proj_splits_,
                                                 proj_rows_per_split_, b.proj_partial)));
        }
        if (!proj_direct) {
            // relation gradients and the sum of the projection gradient's row splits; completes the partial dense gradient
            const size_t proj_total = (size_t)cfg_.n_net() * proj_elems_;
            const unsigned proj_blocks = proj_total ? (unsigned)std::min<size_t>((proj_total + 511) / 512, 148 * 4) : 0;
            if (vec)
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<4>, dim3(n_rel + proj_blocks), dim3(64 * kRelationLanes), 0, stream_,
                                                b.d_relrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, (int)cfg_.n_net(), proj_splits_,
                                                proj_elems_, b.dense_dst, (int)cfg_.world, sync, (int)XCHG_DENSE_PARTIALS, 0)));
            else
                KGE_LAUNCH("dense_partial", KGE_CUDA(launch_dependent(k_dense_partial<1>, dim3(n_rel + proj_blocks), dim3(64 * kRelationLanes), 0, stream_,
                                                b.d_relrow, d_rel_perm_ + sidx * B, d_rel_off_ + sidx * (n_rel + 1), (int)n_rel,
                                                (int)D, b.proj_partial, (int)cfg_.n_net(), proj_splits_,
                                                proj_elems_, b.dense_dst, (int)cfg_.world, sync, (int)XCHG_DENSE_PARTIALS, 0)));
        }
    }
    shards_join();
    if (proj_direct && (side_streams_ & 1u)) side_join(0);  // the relation rows of the partial dense gradient are in place
    KGE_CUDA(cudaGetLastError());
    if (gather_ahead && !gather_beside) launch_gather(step + 1, stream_);  // runs while the partial dense gradients travel

    // 5c. dense parameters: reduce over shards, Adam on the owned slice, publish
    launch_dense_update(step);
    KGE_CUDA(cudaGetLastError());
    if (gather_beside) side_join(1);
}

// ---------------------------------------------------------------------------
// Table and variable I/O

// rows x row_bytes from device memory (rows src_pitch apart) into the caller's contiguous array, in pieces: while one
// piece crosses the link the previous one is copied out of pinned memory (1.4 MB: 180 us as a plain pageable copy, 70 us).
void Engine::copy_out(void* dst, const void* src, size_t src_pitch, size_t row_bytes, size_t rows) {
    if (src_pitch == row_bytes) row_bytes *= rows, rows = 1;
    const size_t per_row = rows == 1 ? kIoPiece : std::max<size_t>(1, (kIoPiece - 256) / row_bytes);  // bytes of one long row, or rows, per piece
    const size_t total = rows == 1 ? row_bytes : rows;
    const size_t piece_bytes = rows == 1 ? kIoPiece : round_up(per_row * row_bytes, 256);
    const PinnedBlock block(piece_bytes * kIoSlots);
    const size_t pieces = (total + per_row - 1) / per_row;
    HostTeam* const team = team_for(total * (rows == 1 ? 1 : row_bytes));
    size_t issued = 0;
    auto issue = [&](size_t i) {
        uint8_t* slot = block.data() + (i % kIoSlots) * piece_bytes;
        const uint8_t* from = static_cast<const uint8_t*>(src) + i * per_row * (rows == 1 ? 1 : src_pitch);
        const size_t count = std::min(per_row, total - i * per_row);
        if (rows == 1) KGE_CUDA(cudaMemcpyAsync(slot, from, count, cudaMemcpyDeviceToHost, stream_));
        else KGE_CUDA(cudaMemcpy2DAsync(slot, row_bytes, from, src_pitch, row_bytes, count, cudaMemcpyDeviceToHost, stream_));
        KGE_CUDA(cudaEventRecord(io_event(i), stream_));
    };
    for (size_t i = 0; i < pieces; ++i) {
        for (; issued < pieces && issued < i + kIoSlots; ++issued) issue(issued);
        KGE_CUDA(cudaEventSynchronize(io_event(i)));
        const size_t unit = rows == 1 ? 1 : row_bytes, count = std::min(per_row, total - i * per_row);
        team_copy(team, static_cast<uint8_t*>(dst) + i * per_row * unit, block.data() + (i % kIoSlots) * piece_bytes, count * unit);
    }
}

// The other way.  Returns when the transfers are complete.
void Engine::copy_in(void* dst, size_t dst_pitch, const void* src, size_t row_bytes, size_t rows) {
    if (dst_pitch == row_bytes) row_bytes *= rows, rows = 1;
    const size_t per_piece = rows == 1 ? kIoPiece : std::max<size_t>(1, (kIoPiece - 256) / row_bytes), total = rows == 1 ? row_bytes : rows;
    const size_t unit = rows == 1 ? 1 : row_bytes, piece_bytes = round_up(per_piece * unit, 256);
    HostTeam* const team = team_for(total * unit);
    const PinnedBlock block(piece_bytes * kIoSlots);
    for (size_t i = 0, at = 0; at < total; ++i, at += per_piece) {
        uint8_t* slot = block.data() + (i % kIoSlots) * piece_bytes;
        const size_t count = std::min(per_piece, total - at);
        if (i >= kIoSlots) KGE_CUDA(cudaEventSynchronize(io_event(i)));
        team_copy(team, slot, static_cast<const uint8_t*>(src) + at * unit, count * unit);
        if (rows == 1) KGE_CUDA(cudaMemcpyAsync(static_cast<uint8_t*>(dst) + at, slot, count, cudaMemcpyHostToDevice, stream_));
        else KGE_CUDA(cudaMemcpy2DAsync(static_cast<uint8_t*>(dst) + at * dst_pitch, dst_pitch, slot, row_bytes, row_bytes, count, cudaMemcpyHostToDevice, stream_));
        KGE_CUDA(cudaEventRecord(io_event(i), stream_));
    }
    KGE_CUDA(cudaStreamSynchronize(stream_));
}

cudaEvent_t Engine::io_event(size_t piece) {
    cudaEvent_t& e = ev_io_[piece % kIoSlots];
    if (!e) KGE_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return e;
}

// Whole rows in the host's element type: `per_shard` rows of every local shard, named by h_idx [n_local, per_shard] or
// (null) the rows first, first + 1, ...  A piece is converted on the GPU, crosses the link and is copied to the caller,
// each while the next one does the step before.  Pieces up to 64 KB are written by the kernel straight into pinned
// memory: that saves a transfer's start but moves only 12 GB/s (the copy engine 45).
void Engine::read_rows(const uint32_t* h_idx, uint32_t first, size_t per_shard, int dtype, void* out) {
    const size_t W = cfg_.row_width(), row_out = W * (dtype == KGE_F32 ? 4 : 2), total = n_local_ * per_shard;
    if (!total) return;
    const size_t per_piece = std::max<size_t>(1, (kIoPiece - 512) / (row_out + 4)), idx_bytes = round_up(per_piece * 4, 256);
    const size_t piece_bytes = idx_bytes + round_up(per_piece * row_out, 256), pieces = (total + per_piece - 1) / per_piece;
    const PinnedBlock block(piece_bytes * kIoSlots);
    HostTeam* const team = team_for(total * row_out);
    DeviceBlock staging;
    size_t issued = 0;
    for (size_t i = 0; i < pieces; ++i) {
        for (; issued < pieces && issued < i + kIoSlots; ++issued) {
            uint8_t* slot = block.data() + (issued % kIoSlots) * piece_bytes;
            const size_t at = issued * per_piece, count = std::min(per_piece, total - at);
            uint32_t* idx = nullptr;
            if (h_idx) {
                idx = reinterpret_cast<uint32_t*>(slot);
                std::memcpy(idx, h_idx + at, count * 4);
            }
            const RowSource rows{shards_[0].table, table_stride_, idx, first, at, per_shard};
            const unsigned grid = (unsigned)count;
            const bool staged = count * row_out > kIoDirectBytes && piece_bytes <= kIoPiece;
            uint8_t* to = staged ? staging.get() + (issued % kIoSlots) * kIoPiece : slot + idx_bytes;
            if (dtype == KGE_F32)
                KGE_DISPATCH_ROW(cfg_, k_read_rows<ST, FT, float><<<grid, 128, 0, stream_>>>(rows, layout_, reinterpret_cast<float*>(to)));
            else
                k_read_rows<__half, __half, __half><<<grid, 128, 0, stream_>>>(rows, layout_, reinterpret_cast<__half*>(to));
            KGE_CUDA(cudaGetLastError());
            if (staged) KGE_CUDA(cudaMemcpyAsync(slot + idx_bytes, to, count * row_out, cudaMemcpyDeviceToHost, stream_));
            KGE_CUDA(cudaEventRecord(io_event(issued), stream_));
        }
        if (team && i == 0) team_touch(*team, out, total * row_out);
        KGE_CUDA(cudaEventSynchronize(io_event(i)));
        const size_t at = i * per_piece;
        team_copy(team, static_cast<uint8_t*>(out) + at * row_out, block.data() + (i % kIoSlots) * piece_bytes + idx_bytes, std::min(per_piece, total - at) * row_out);
    }
}

// The other way: fresh rows with the given features (as "write_entity"), or whole rows.
void Engine::write_rows(const uint32_t* h_idx, uint32_t first, size_t per_shard, int dtype, const void* data, bool whole_rows) {
    const size_t per_row = whole_rows ? cfg_.row_width() : cfg_.f, row_in = per_row * (dtype == KGE_F32 ? 4 : 2), total = n_local_ * per_shard;
    if (!total) return;
    const size_t per_piece = std::max<size_t>(1, (kIoPiece - 256) / std::max<size_t>(row_in, 64)), piece_bytes = round_up(per_piece * row_in, 256);
    const PinnedBlock block(piece_bytes * kIoSlots);
    HostTeam* const team = team_for(total * row_in);
    DeviceBlock staging;
    const float stddev = cfg_.init_scale / (float)cfg_.d;  // src/poplar_kge.cpp:865
    if (h_idx) copy_in(d_rw_idx_, total * 4, h_idx, total * 4, 1);  // all of them: a slot looks for later ones with its row
    for (size_t i = 0, at = 0; at < total; ++i, at += per_piece) {
        uint8_t* slot = block.data() + (i % kIoSlots) * piece_bytes;
        const size_t count = std::min(per_piece, total - at);
        if (i >= kIoSlots) KGE_CUDA(cudaEventSynchronize(io_event(i)));
        if (row_in) team_copy(team, slot, static_cast<const uint8_t*>(data) + at * row_in, count * row_in);
        const RowSource rows{shards_[0].table, table_stride_, h_idx ? d_rw_idx_ + at : nullptr, first, at, per_shard};
        const unsigned grid = (unsigned)count;
        if (count * row_in > kIoDirectBytes && piece_bytes <= kIoPiece) {  // shorter pieces are read by the kernel across the link
            uint8_t* to = staging.get() + (i % kIoSlots) * kIoPiece;
            KGE_CUDA(cudaMemcpyAsync(to, slot, count * row_in, cudaMemcpyHostToDevice, stream_));
            slot = to;
        }
        if (dtype == KGE_F32) {
            using IT = float;
            if (whole_rows) KGE_DISPATCH_ROW(cfg_, k_write_rows<ST, FT, IT><<<grid, 128, 0, stream_>>>(rows, layout_, (const IT*)slot));
            else KGE_DISPATCH_ROW(cfg_, k_write_entity<ST, FT, IT><<<grid, 128, 0, stream_>>>(rows, layout_, (const IT*)slot, cfg_.seed, shard0_, stddev));
        } else {
            using IT = __half;
            if (whole_rows) KGE_DISPATCH_ROW(cfg_, k_write_rows<ST, FT, IT><<<grid, 128, 0, stream_>>>(rows, layout_, (const IT*)slot));
            else KGE_DISPATCH_ROW(cfg_, k_write_entity<ST, FT, IT><<<grid, 128, 0, stream_>>>(rows, layout_, (const IT*)slot, cfg_.seed, shard0_, stddev));
        }
        KGE_CUDA(cudaGetLastError());
        KGE_CUDA(cudaEventRecord(io_event(i), stream_));
    }
    KGE_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::cmd_read_entity(std::vector<HostArray>& arrays) {
    const size_t n = n_local_, rw = cfg_.rw_batch, W = cfg_.row_width();
    HostArray& idx = find_array(arrays, "read_indices", KGE_U32, {n, rw});
    const int out_dtype = cfg_.state_type == ST_F32 ? KGE_F32 : KGE_F16;
    HostArray& out = find_array(arrays, "read_data", out_dtype, {n, rw, W});
    const uint32_t* h = static_cast<const uint32_t*>(idx.data);
    for (size_t i = 0; i < n * rw; ++i)
        if (h[i] >= cfg_.n_entity)
            fail(KGE_INVALID_ARGUMENT, msg() << "'read_indices' holds index " << h[i] << ", not below model.n_entity ("
                                             << cfg_.n_entity << ")");
    read_rows(h, 0, rw, out_dtype, out.data);
}

// "read_entity_range" / "write_entity_range": what "read_entity" / "write_entity" do to the rows `row_range` u32 [2] =
// (first, count) of every local shard, whatever rw_batch_size: read_data [n, count, 3D+F] in the state type;
// write_features [n, count, F], float32 or float16.
void Engine::cmd_entity_range(std::vector<HostArray>& arrays, bool read) {
    HostArray& range = find_array(arrays, "row_range", KGE_U32, {2});
    const size_t n = n_local_, first = static_cast<const uint32_t*>(range.data)[0], count = static_cast<const uint32_t*>(range.data)[1];
    if (first + count > cfg_.n_entity)
        fail(KGE_INVALID_ARGUMENT, msg() << "'row_range' covers rows [" << first << ", " << first + count << "), not within model.n_entity (" << cfg_.n_entity << ")");
    if (read) {
        const int out_dtype = cfg_.state_type == ST_F32 ? KGE_F32 : KGE_F16;
        HostArray& out = find_array(arrays, "read_data", out_dtype, {n, count, cfg_.row_width()});
        return read_rows(nullptr, (uint32_t)first, count, out_dtype, out.data);
    }
    HostArray* data = nullptr;
    for (HostArray& a : arrays)
        if (a.name == "write_features") data = &a;
    if (!data) fail(KGE_INVALID_ARGUMENT, "Key not found 'write_features'");
    find_array(arrays, "write_features", data->dtype == KGE_F16 ? KGE_F16 : KGE_F32, {n, count, cfg_.f});
    write_rows(nullptr, (uint32_t)first, count, data->dtype, data->data, false);
}

// "dump_entity_rows" / "restore_entity_rows": a contiguous range of one local shard's table as it
// is stored (no type conversion, optimiser state included), for checkpoints of tables too large
// to pass through host arrays of the state type at once.  `shard_range` u32 [3] = (local shard,
// first row, row count); `rows` u32 [row count, row bytes / 4].  The reference reads and writes
// the table only through indexed chunks of rw_batch_size rows (src/poplar_kge.cpp:857-871;
// read_entity_all, src/python/poplar_kge.py:583-598); a stored range is one plain copy.
void Engine::cmd_copy_entity_range(std::vector<HostArray>& arrays, bool to_host) {
    HostArray& range = find_array(arrays, "shard_range", KGE_U32, {3});
    const uint32_t* r = static_cast<const uint32_t*>(range.data);
    const size_t shard = r[0], first = r[1], count = r[2];
    if (shard >= n_local_) fail(KGE_INVALID_ARGUMENT, msg() << "'shard_range' names local shard " << shard << " of " << n_local_);
    if (first + count > cfg_.n_entity)
        fail(KGE_INVALID_ARGUMENT, msg() << "'shard_range' covers rows [" << first << ", " << first + count
                                         << "), not within model.n_entity (" << cfg_.n_entity << ")");
    HostArray& rows = find_array(arrays, "rows", KGE_U32, {count, (size_t)layout_.row_bytes / 4});
    if (!count) return;
    unsigned char* table = shards_[shard].table + first * (size_t)layout_.row_bytes;
    const size_t bytes = count * (size_t)layout_.row_bytes;
    if (to_host)
        KGE_CUDA(cudaMemcpyAsync(rows.data, table, bytes, cudaMemcpyDeviceToHost, stream_));
    else
        KGE_CUDA(cudaMemcpyAsync(table, rows.data, bytes, cudaMemcpyHostToDevice, stream_));
    KGE_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::cmd_write_entity(std::vector<HostArray>& arrays, bool whole_rows) {
    const size_t n = n_local_, rw = cfg_.rw_batch, W = cfg_.row_width(), F = cfg_.f;
    HostArray& idx = find_array(arrays, "write_indices", KGE_U32, {n, rw});
    const char* data_name = whole_rows ? "write_data" : "write_features";
    const std::vector<size_t> shape = {n, rw, whole_rows ? W : F};
    // The host array is in the state type (the reference's single dtype); a float16 array is
    // also taken for features when they are stored as float16.
    HostArray* data = nullptr;
    for (HostArray& a : arrays)
        if (a.name == data_name) data = &a;
    if (!data) fail(KGE_INVALID_ARGUMENT, msg() << "Key not found '" << data_name << "'");
    const int state_dtype = cfg_.state_type == ST_F32 ? KGE_F32 : KGE_F16;
    const bool f16_features_ok = !whole_rows && cfg_.feature_type == ST_F16 && data->dtype == KGE_F16;
    find_array(arrays, data_name, f16_features_ok ? KGE_F16 : state_dtype, shape);
    const uint32_t* h = static_cast<const uint32_t*>(idx.data);
    for (size_t i = 0; i < n * rw; ++i)
        if (h[i] >= cfg_.n_entity)
            fail(KGE_INVALID_ARGUMENT, msg() << "'write_indices' holds index " << h[i] << ", not below model.n_entity ("
                                             << cfg_.n_entity << ")");
    write_rows(h, 0, rw, data->dtype, data->data, whole_rows);
}

void Engine::cmd_initialise_entities() {
    const float stddev = cfg_.init_scale / (float)cfg_.d;
    for (unsigned l = 0; l < n_local_; ++l) {
        KGE_DISPATCH_ROW(cfg_, k_init_table<ST, FT><<<148 * 8, 256, 0, stream_>>>(shards_[l].table, layout_, (size_t)cfg_.n_entity,
                                                                               cfg_.seed, shard0_ + l, stddev));
    }
    KGE_CUDA(cudaGetLastError());
    KGE_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::cmd_read_write_variable(std::vector<HostArray>& arrays, const std::string& name, bool write) {
    const Variable* var = nullptr;
    for (const Variable& v : variables_)
        if (v.name == name) var = &v;
    if (!var) fail(KGE_INVALID_ARGUMENT, msg() << "Key not found '" << name << "'");
    HostArray& value = find_array(arrays, "value", var->dtype, var->shape);
    if (var->kind == 3) {  // step: one counter, presented per shard
        uint32_t* p = static_cast<uint32_t*>(value.data);
        if (write) {
            for (unsigned s = 1; s < cfg_.n_shard; ++s)
                if (p[s] != p[0]) fail(KGE_INVALID_ARGUMENT, "'step' must hold the same value for every shard");
            step_ = p[0];
        } else {
            for (unsigned s = 0; s < cfg_.n_shard; ++s) p[s] = (uint32_t)step_;
        }
        return;
    }
    const size_t count = value.count();
    if (count == 0) return;
    float* base = var->kind == 0 ? dense_ : var->kind == 1 ? dense_m_ : dense_v_;
    // Rows of the dense vector are d floats wide; a variable may show fewer columns of them to the
    // host (RotatE's angles are the first half of their rows).
    const size_t D = cfg_.d, row0 = var->offset / D, W = cfg_.world;
    const size_t cols = var->flat ? D : var->shape[1], n_rows = var->flat ? count / D : var->shape[0];
    float* host = static_cast<float*>(value.data);
    if (write) {
        // on the engine's stream, so that the kernel that derives the lower plane is ordered behind the copy
        copy_in(base + var->offset, D * 4, host, cols * 4, n_rows);
        if (var->kind == 0) refresh_lower_plane(var->offset, n_rows * D);
        return;
    }
    if (var->kind == 0 || cfg_.world == 1) {
        copy_out(host, base + var->offset, D * 4, cols * 4, n_rows);
        return;
    }
    KGE_CUDA(cudaStreamSynchronize(stream_));
    // Optimiser state lives with the process that owns the row (src/poplar_kge.cpp:329-339): row r of
    // the dense vector with process r % world.  Collect each owner's rows through its mapped arena.
    for (size_t p = 0; p < W; ++p) {
        const size_t first = row0 + (p + W - row0 % W) % W;
        if (first >= row0 + n_rows) continue;
        const size_t rows = (row0 + n_rows - first + W - 1) / W;
        const float* src = (const float*)(peer_arena_[p] + arena_offset_dense(var->kind)) + first * D;
        KGE_CUDA(cudaMemcpy2D(host + (first - row0) * cols, W * cols * 4, src, W * D * 4, cols * 4, rows, cudaMemcpyDeviceToHost));
    }
}

// The projections are tensor-core operands: their lower TF32 plane follows every change of the values.
void Engine::refresh_lower_plane(size_t offset, size_t count) {
    if (!planes_ || count == 0) return;
    k_lower_plane<<<(unsigned)std::min<size_t>((count + 255) / 256, 148 * 8), 256, 0, stream_>>>(dense_ + offset, count, dense_lo_ + offset);
    KGE_CUDA(cudaGetLastError());
    KGE_CUDA(cudaStreamSynchronize(stream_));
}

// Where a pass has a wave of 128 x 128 tiles its contractions run on float16 planes (tc::HalfRows): the fp16 features as
// they lie in the table, everything else in two parts, half the instructions and bytes of the TF32 planes and no copy of
// the features.  Smaller passes divide k over a cluster, which those instantiations do not.  A pass of 18944 rows and
// 1250 queries, d 256, f 768: 308 us on TF32 planes, 120 us.
static bool fills_gpu(unsigned m, unsigned n) { return ceil_div(m, 128) * ceil_div(n, 128) >= 148; }

void Engine::ensure_predict_buffers() {
    if (p_raw_) return;
    const size_t Q = (size_t)cfg_.n_shard * cfg_.predict_hr, D = cfg_.d;
    p_head_hidden_ = (float*)device_alloc((size_t)cfg_.predict_hr * D * 4);
    // L1 has no contraction form; everything else ranks with the plane-fed tensor-core kernel
    predict_planes_ = planes_ && cfg_.dist_fn != DIST_L1 && cfg_.score_fn != SCORE_TRANSH;
    // Rows per pass over the table.  On the tensor cores: 148 tiles of 128 rows, so that the hidden
    // rows' contraction (2 column tiles) and the scores' (10 query tiles at 1250 queries) both fill
    // whole waves of 148 blocks.
    // Elsewhere as many as 64 MB of scores hold, between 4096 and 65536: few queries make short kernels.
    predict_chunk_ = predict_planes_ ? 148u * 128u : (unsigned)std::min<size_t>(65536, std::max<size_t>(4096, ((size_t)16 << 20) / Q / 128 * 128));
    predict_chunk_ = std::min(predict_chunk_, (unsigned)round_up(cfg_.n_entity, 128));
    if (const char* v = std::getenv("KGE_PREDICT_PASS_ROWS")) predict_chunk_ = std::max(64u, (unsigned)std::atoi(v) / 4u * 4u);
    if (cfg_.score_fn == SCORE_TRANSH) predict_chunk_ = std::min(predict_chunk_, (unsigned)kTranshMaxTails);
    p_chunk_hidden_ = (float*)device_alloc((size_t)predict_chunk_ * D * 4);
    p_raw_ = (float*)device_alloc(Q * predict_chunk_ * 4);
    if (predict_planes_) {
        p_chunk_lo_ = (float*)device_alloc((size_t)predict_chunk_ * D * 4);
        p_query_lo_ = (float*)device_alloc(Q * D * 4);
        if (cfg_.f) p_feat_ = (float*)device_alloc((size_t)predict_chunk_ * feat_stride_ * 4);
        p_half_stride_ = (int)round_up(D, 8);
        p_half_q_ = (__half*)device_alloc(2 * Q * p_half_stride_ * sizeof(__half));
        p_half_q_info_ = (float2*)device_alloc(Q * sizeof(float2));
        p_half_t_ = (__half*)device_alloc(2 * (size_t)predict_chunk_ * p_half_stride_ * sizeof(__half));
        p_half_t_info_ = (float2*)device_alloc(predict_chunk_ * sizeof(float2));
        if (cfg_.f && cfg_.feature_type == ST_F16) {
            p_half_w_ = (__half*)device_alloc(2 * (size_t)cfg_.f * p_half_stride_ * sizeof(__half));
            p_half_w_info_ = (float2*)device_alloc(D * sizeof(float2));
        }
    }
    if (mlp_on()) {
        const size_t rows = std::max<size_t>(cfg_.predict_hr, predict_chunk_);
        p_mlp_cat_ = (float*)device_alloc(rows * 2 * D * 4);
        p_mlp_pre_ = (float*)device_alloc(rows * cfg_.mlp * 4);
        p_mlp_out_ = (float*)device_alloc(rows * D * 4);
    }
    p_cand_ = (unsigned long long*)device_alloc(Q * kTopkCandidates * sizeof(unsigned long long));
    p_cand_count_ = (int*)device_alloc(Q * sizeof(int));
    KGE_CUDA(cudaMemset(p_cand_count_, 0, Q * sizeof(int)));
    d_iota_ = (uint32_t*)device_alloc((size_t)cfg_.predict_hr * 4);
    std::vector<uint32_t> iota(cfg_.predict_hr);
    for (unsigned i = 0; i < cfg_.predict_hr; ++i) iota[i] = i;
    KGE_CUDA(cudaMemcpy(d_iota_, iota.data(), iota.size() * 4, cudaMemcpyHostToDevice));
    for (ShardBuffers& b : shards_) {
        b.topk_state = (unsigned long long*)device_alloc(Q * kTopkCapacity * sizeof(unsigned long long));
        b.topk_count = (int*)device_alloc(Q * sizeof(int));
    }
}

// Merges the scores of rows start .. start + c - 1 (in p_raw_) into every query's best list: the filter at
// full bandwidth, then one warp per query on what it left.
void Engine::launch_topk(ShardBuffers& b, unsigned c, uint32_t start, uint32_t last, const TopkParams& tp, bool filtered) {
    const unsigned Q = (unsigned)tp.n_query;
    if (start == 1) {  // nothing ranked yet: parts of at least 512 scores, as many lists as the candidates have room for
        const unsigned parts = std::max(1u, std::min({(unsigned)kTopkCandidates / (unsigned)tp.n_best, ceil_div(c, 512u), 64u}));
        const auto seed = tp.n_best <= 32 ? k_topk_seed<true> : k_topk_seed<false>;
        KGE_LAUNCH("predict_topk", seed<<<dim3(ceil_div(Q, 4), parts), 128, 0, stream_>>>(p_raw_, (int)c, start, last, p_cand_, p_cand_count_, tp));
    } else if (!filtered) {  // else the score kernel's epilogue has left the candidates
        const dim3 fgrid(std::max(1u, std::min(ceil_div(c, 4 * 256), 8u)), Q);
        KGE_LAUNCH("predict_topk", k_topk_filter<<<fgrid, 256, 0, stream_>>>(p_raw_, (int)c, start, last, b.topk_state, b.topk_count, p_cand_, p_cand_count_, tp));
    }
    // On the tensor cores the merge (13 us for 1250 queries) runs beside the next pass's hidden rows, which it has nothing
    // to do with; the next scores wait for it (join_topk).
    const cudaStream_t st = predict_planes_ ? side_begin() : stream_;
    KGE_LAUNCH("predict_topk", k_topk_update<<<ceil_div(Q, 4), 128, 0, st>>>(p_raw_, (int)c, start, last, b.topk_state, b.topk_count, tp, p_cand_,
                                                                            p_cand_count_));
    if (predict_planes_) side_end(0);
    topk_beside_ = predict_planes_;
}

void Engine::join_topk() {
    if (topk_beside_) side_join(0);
    topk_beside_ = false;
}

// Ranks every real row of the local shards as a tail for the queries of all shards
// (src/poplar_kge.cpp:812-855): predicted tails of the local queries are written into every
// process's query buffer (the all-gather of :825-828); each local shard then streams its table in
// batches, scores them and keeps the n_best per query; the results go back to the asking shard's
// process (the two all-to-alls of :847-850).
void Engine::cmd_predict(std::vector<HostArray>& arrays) {
    const size_t n = n_local_, hr = cfg_.predict_hr, nb = cfg_.predict_n_best, D = cfg_.d;
    const size_t Q = (size_t)cfg_.n_shard * hr;
    HostArray& head = find_array(arrays, "predict_head", KGE_U32, {n, hr});
    HostArray& relation = find_array(arrays, "predict_relation", KGE_U32, {n, hr});
    HostArray& count = find_array(arrays, "predict_entity_count", KGE_U32, {n});
    HostArray& scores = find_array(arrays, "predict_scores", KGE_F32, {n, cfg_.n_shard, hr, nb});
    HostArray& indices = find_array(arrays, "predict_indices", KGE_U32, {n, cfg_.n_shard, hr, nb});
    if (hr == 0) fail(KGE_INVALID_ARGUMENT, "'execution.predict_hr_batch_size' must be positive to rank queries");
    if (nb == 0 || nb > kTopkCapacity / 2)
        fail(KGE_INVALID_ARGUMENT, msg() << "'execution.predict_n_best' must be between 1 and " << kTopkCapacity / 2);
    if (!connected_) fail(KGE_LOGIC_ERROR, "world_size > 1 but kge_comm_connect has not been called");
    require_usable();
    const uint32_t* h_head = static_cast<const uint32_t*>(head.data);
    const uint32_t* h_rel = static_cast<const uint32_t*>(relation.data);
    const uint32_t* h_count = static_cast<const uint32_t*>(count.data);
    for (size_t i = 0; i < n * hr; ++i) {
        if (h_head[i] >= cfg_.n_entity)
            fail(KGE_INVALID_ARGUMENT, msg() << "'predict_head' holds index " << h_head[i] << ", not below model.n_entity (" << cfg_.n_entity << ")");
        if (h_rel[i] >= cfg_.n_relation_type)
            fail(KGE_INVALID_ARGUMENT, msg() << "'predict_relation' holds index " << h_rel[i] << ", not below model.n_relation_type (" << cfg_.n_relation_type << ")");
    }
    for (size_t l = 0; l < n; ++l)
        if (h_count[l] >= cfg_.n_entity)
            fail(KGE_INVALID_ARGUMENT, msg() << "'predict_entity_count' (" << h_count[l] << ") must be below model.n_entity (" << cfg_.n_entity << ")");
    ensure_predict_buffers();
    KGE_CUDA(cudaStreamSynchronize(stream_));
    uint32_t* d_head = d_rw_idx_;
    uint32_t* d_rel = d_rw_idx_ + n * hr;
    KGE_CUDA(cudaMemcpyAsync(d_head, h_head, n * hr * 4, cudaMemcpyHostToDevice, stream_));
    KGE_CUDA(cudaMemcpyAsync(d_rel, h_rel, n * hr * 4, cudaMemcpyHostToDevice, stream_));
    unsigned longest = 0;  // rows of the command's longest pass
    for (unsigned l = 0; l < n; ++l) longest = std::max(longest, (unsigned)std::min<uint32_t>(predict_chunk_, h_count[l]));

    const bool two_nets = cfg_.n_net() == 2, vec = (D % 4) == 0;
    const float* W_head = cfg_.n_net() >= 1 ? dense_ + dense_bounds_[1] : nullptr;
    const float* W_tail = two_nets ? dense_ + dense_bounds_[2] : W_head;
    const unsigned dtiles = ceil_div((unsigned)D, 64);
    launch_counter_ = 0;
    const bool half_projection = predict_planes_ && p_half_w_ && fills_gpu(longest, (unsigned)D);
    if (half_projection) {
        KGE_CUDA(cudaMemsetAsync(d_planes_short_, 0, 4, stream_));
        KGE_LAUNCH("predict_planes", tc::k_half_columns<<<ceil_div((unsigned)D, 32), 256, 0, stream_>>>(
                                         W_tail, (int)cfg_.f, (int)D, p_half_stride_, p_half_w_, p_half_w_ + (size_t)cfg_.f * p_half_stride_, p_half_w_info_, d_planes_short_));
        KGE_CUDA(cudaGetLastError());
        KGE_CUDA(cudaMemcpyAsync(pinned_ + status_at_ + 2, d_planes_short_, 4, cudaMemcpyDeviceToHost, stream_));
        KGE_CUDA(cudaEventRecord(io_event(0), stream_));
    }

    // 1. predicted tails of the local queries, written into every process's gathered query buffer: from the table itself
    // without features, all shards at once, else from the hidden rows of one shard after the other
    const bool from_table = cfg_.f == 0;
    const unsigned at_once = from_table ? (unsigned)kShardBatch : 1u;
    const int value_type = !from_table ? 0 : cfg_.value_bf16 ? 2 : cfg_.state_type == ST_F16 ? 1 : 0;
    for (unsigned l0 = 0; l0 < n; l0 += at_once) {
        const unsigned count_l = std::min<unsigned>(at_once, (unsigned)n - l0);
        if (!from_table) {
            dim3 grid(ceil_div((unsigned)hr, 64), dtiles, 1);
            KGE_LAUNCH("predict_hidden", KGE_DISPATCH_ROW(cfg_, k_hidden<ST, FT><<<grid, 256, 0, stream_>>>(
                                                                    shards_[l0].table, layout_, d_head + l0 * hr, 0u, (int)hr, W_head,
                                                                    nullptr, p_head_hidden_, nullptr)));
            if (mlp_on()) launch_mlp_forward(shards_[l0].table, d_head + l0 * hr, 0u, (unsigned)hr, 0, p_head_hidden_, p_mlp_cat_, p_mlp_pre_, p_mlp_out_);
        }
        for (unsigned p = 0; p < cfg_.world; ++p) {
            ShardArgs<LookupArgs> query{};
            for (unsigned i = 0; i < count_l; ++i) {
                const unsigned l = l0 + i;
                LookupArgs& a = query.s[i];
                a.rows = from_table ? LookupRows{shards_[l].table, nullptr, d_head + l * hr, nullptr, layout_.row_bytes}
                                    : LookupRows{reinterpret_cast<const uint8_t*>(p_head_hidden_), nullptr, d_iota_, nullptr, D * 4};
                a.relation = d_rel + l * hr;
                a.pred = (float*)(peer_arena_[p] + arena_offset_predict(0)) + (size_t)(shard0_ + l) * hr * D;
                a.nrm = a.pred + Q * D;  // TransH
            }
            LookupSizes sizes{};
            sizes.rel_table = dense_;
            sizes.normal_table = dense_ + dense_bounds_[3];
            sizes.B = (int)hr;
            sizes.D = (int)D;
            KGE_LAUNCH("predict_query", KGE_CUDA(kge::launch_lookup(query, (int)count_l, sizes, cfg_.score_fn, value_type, stream_)));
        }
    }
    KGE_CUDA(cudaGetLastError());
    launch_barrier();

    // 2. stream each local shard's rows past all queries
    const float* queries = (const float*)(arena_ + arena_offset_predict(0));
    if (half_projection) KGE_CUDA(cudaEventSynchronize(io_event(0)));  // the queries are being prepared meanwhile
    p_half_w_usable_ = half_projection && pinned_[status_at_ + 2] == 0;
    if (predict_planes_) {
        KGE_LAUNCH("predict_planes", k_lower_plane<<<(unsigned)std::min<size_t>((Q * D + 255) / 256, 148 * 8), 256, 0, stream_>>>(queries, Q * D, p_query_lo_));
        if (fills_gpu((unsigned)Q, longest)) KGE_LAUNCH("predict_planes", tc::k_half_rows<<<ceil_div((unsigned)Q, 8), 256, 0, stream_>>>(queries, (int)Q, (int)D, p_half_stride_, p_half_q_,
                                                                                                    p_half_q_ + Q * p_half_stride_, p_half_q_info_));
    }
    TopkParams tp{(int)Q, (int)nb, score_is_gamma_minus_distance(cfg_.score_fn) ? 1 : 0, cfg_.gamma};
    for (unsigned l = 0; l < n; ++l) {
        ShardBuffers& b = shards_[l];
        KGE_CUDA(cudaMemsetAsync(b.topk_count, 0, Q * sizeof(int), stream_));
        const uint32_t last = h_count[l];
        for (uint32_t start = 1; start <= last; start += predict_chunk_) {
            const unsigned c = std::min<uint32_t>(predict_chunk_, last - start + 1);
            if (predict_planes_) {
                const bool filtered = predict_pass_planes(b, start, c, last, tp, queries, (unsigned)Q, W_tail == W_head ? 0 : 1);
                launch_topk(b, c, start, last, tp, filtered);
                continue;
            }
            dim3 hgrid(ceil_div(c, 64), dtiles, 1);
            KGE_LAUNCH("predict_hidden", KGE_DISPATCH_ROW(cfg_, k_hidden<ST, FT><<<hgrid, 256, 0, stream_>>>(
                                                                    b.table, layout_, nullptr, start, (int)c, W_tail, nullptr,
                                                                    p_chunk_hidden_, nullptr)));
            if (mlp_on()) launch_mlp_forward(b.table, nullptr, start, c, two_nets ? 1 : 0, p_chunk_hidden_, p_mlp_cat_, p_mlp_pre_, p_mlp_out_);
            if (cfg_.score_fn == SCORE_TRANSH) {
                KGE_LAUNCH("predict_score", KGE_CUDA(launch_transh_score(queries, queries + Q * D, p_chunk_hidden_, p_raw_, (int)Q, (int)c, (int)D, stream_)));
            } else
            KGE_LAUNCH("predict_score", KGE_CUDA(launch_score(cfg_.dist_fn, queries, p_chunk_hidden_, p_raw_, (int)Q, (int)c, (int)D, stream_)));
            launch_topk(b, c, start, last, tp, false);
        }
        join_topk();
        KGE_LAUNCH("predict_finish", k_topk_finish<<<(unsigned)Q, 128, 0, stream_>>>(
                                         b.topk_state, b.topk_count, (int)Q, (int)hr, (int)nb, b.predict_score_dst,
                                         b.predict_index_dst));
        KGE_CUDA(cudaGetLastError());
    }
    launch_barrier();
    const size_t result_bytes = n * cfg_.n_shard * hr * nb * 4, slot = round_up(result_bytes, 256);
    if (2 * slot + 256 <= PinnedPool::kBlock) {  // results and status words in one wait
        const PinnedBlock block;
        KGE_CUDA(cudaMemcpyAsync(block.data(), arena_ + arena_offset_predict(1), slot + result_bytes, cudaMemcpyDeviceToHost, stream_));
        check_device_status();
        std::memcpy(scores.data, block.data(), result_bytes);
        std::memcpy(indices.data, block.data() + slot, result_bytes);
    } else {
        copy_out(scores.data, arena_ + arena_offset_predict(1), result_bytes, result_bytes, 1);
        copy_out(indices.data, arena_ + arena_offset_predict(2), result_bytes, result_bytes, 1);
        check_device_status();
    }
    timing_collect();
    last_launches_ = launch_counter_;
}

// One pass of predict on the tensor cores: hidden rows of the table rows [start, start + c) as the
// contraction feature . W + value, then their scores against all Q queries: the dot product, or
// the L2 distance as |q|^2 + |t|^2 - 2 q.t with the direct form where that cancels, so identical
// rows still score identically and an exact match still scores gamma
// (src/poplar_kge.cpp:812-855; src/poplar_extensions/distance.cpp:151-185).
// Returns whether the score kernel has also filtered the pass's scores against the queries' cut-offs
// (the L2 form; dot products leave that to k_topk_filter).
bool Engine::predict_pass_planes(ShardBuffers& b, uint32_t start, unsigned c, uint32_t last, const TopkParams& tp, const float* queries, unsigned Q,
                                 int net) {
    const unsigned D = cfg_.d, F = cfg_.f;
    const uint8_t* rows = b.table + (size_t)start * layout_.row_bytes;
    const bool hidden_half = F > 0 && p_half_w_usable_ && fills_gpu(c, D), score_half = fills_gpu(Q, c);
    auto half_plane = [&](const __half* hi, const __half* lo, bool mn_major) {
        return tc::PlaneOperand{reinterpret_cast<const float*>(hi), reinterpret_cast<const float*>(lo), (long long)p_half_stride_ * 2, mn_major ? 1 : 0, 16};
    };
    if (hidden_half) {
        tc::PlaneProblem p{};
        p.A = tc::PlaneOperand{reinterpret_cast<const float*>(rows + layout_.off_feat), nullptr, (long long)layout_.row_bytes, 0, 16};
        p.B = half_plane(p_half_w_, p_half_w_ + (size_t)F * p_half_stride_, true);
        p.half_b.info = p_half_w_info_;
        p.g.M = (int)c; p.g.N = (int)D; p.g.K = (int)F;
        p.g.epilogue = tc::EPI_ADD_TABLE_VALUE;
        p.g.out = p_chunk_hidden_; p.g.ldc = D; p.g.block_rows = 1;
        p.g.x_base = rows; p.g.x_row_stride_bytes = layout_.row_bytes;
        p.g.x_is_half = cfg_.value_bf16 ? 2 : (cfg_.state_type == ST_F16 ? 1 : 0);
        launch_planes("predict_hidden", &p, 1, tc::SIDE_NONE, -1, -1);
    } else if (F > 0) {
        FeaturePlanes fp{};
        const bool half_features = cfg_.feature_type == ST_F16;
        (half_features ? fp.wide : fp.lo) = p_feat_;
        fp.stride = feat_stride_;
        fp.off_feat = layout_.off_feat;
        const size_t units = (size_t)c * ((layout_.row_bytes - layout_.off_feat) >> 4);
        KGE_LAUNCH("predict_planes", k_table_feature_planes<<<(unsigned)std::min<size_t>((units + 255) / 256, 148 * 16), 256, 0, stream_>>>(
                                         b.table, layout_, start, (int)c, fp));
        tc::PlaneProblem p{};
        p.A = half_features ? tc::PlaneOperand{p_feat_, nullptr, (long long)feat_stride_ * 4, 0, 0}
                            : tc::PlaneOperand{reinterpret_cast<const float*>(rows + layout_.off_feat), p_feat_, (long long)layout_.row_bytes, 0, 0};
        const size_t w = dense_bounds_[1 + net];
        p.B = tc::PlaneOperand{dense_ + w, dense_lo_ + w, (long long)D * 4, 1, 0};
        p.g.M = (int)c; p.g.N = (int)D; p.g.K = (int)F;
        p.g.epilogue = tc::EPI_ADD_TABLE_VALUE;
        p.g.out = p_chunk_hidden_; p.g.ldc = D; p.g.block_rows = 1;
        p.g.x_base = rows; p.g.x_row_stride_bytes = layout_.row_bytes;
        p.g.x_is_half = cfg_.value_bf16 ? 2 : (cfg_.state_type == ST_F16 ? 1 : 0);
        launch_planes("predict_hidden", &p, 1, tc::SIDE_NONE, -1, -1);
    } else {
        dim3 hgrid(ceil_div(c, 64), ceil_div(D, 64), 1);
        KGE_LAUNCH("predict_hidden", KGE_DISPATCH_ROW(cfg_, k_hidden<ST, FT><<<hgrid, 256, 0, stream_>>>(
                                                                b.table, layout_, nullptr, start, (int)c, nullptr, nullptr, p_chunk_hidden_, nullptr)));
    }
    tc::PlaneProblem s{};
    if (score_half) {
        __half* const lo = p_half_t_ + (size_t)predict_chunk_ * p_half_stride_;
        KGE_LAUNCH("predict_planes", tc::k_half_rows<<<ceil_div(c, 8), 256, 0, stream_>>>(p_chunk_hidden_, (int)c, (int)D, p_half_stride_, p_half_t_, lo, p_half_t_info_));
        s.A = half_plane(p_half_q_, p_half_q_ + (size_t)Q * p_half_stride_, false);
        s.B = half_plane(p_half_t_, lo, false);
        s.half_a = tc::HalfRows{p_half_q_info_, queries, (long long)D * 4};
        s.half_b = tc::HalfRows{p_half_t_info_, p_chunk_hidden_, (long long)D * 4};
    } else {
        KGE_LAUNCH("predict_planes", k_lower_plane<<<(unsigned)std::min<size_t>(((size_t)c * D + 255) / 256, 148 * 16), 256, 0, stream_>>>(
                                         p_chunk_hidden_, (size_t)c * D, p_chunk_lo_));
        s.A = tc::PlaneOperand{queries, p_query_lo_, (long long)D * 4, 0, 0};
        s.B = tc::PlaneOperand{p_chunk_hidden_, p_chunk_lo_, (long long)D * 4, 0, 0};
    }
    s.g.M = (int)Q; s.g.N = (int)c; s.g.K = (int)D;
    const bool l2 = cfg_.dist_fn == DIST_L2;
    s.g.epilogue = l2 ? tc::EPI_L2_DISTANCE : tc::EPI_STORE;
    s.g.out = p_raw_; s.g.ldc = c; s.g.block_rows = 1;
    const bool filtered = l2 && filter_in_scores_;
    if (filtered) s.filter = tc::TopkFilterArgs{b.topk_state, b.topk_count, p_cand_, p_cand_count_, start, last, tp.n_best, tp.score_is_gamma_minus, tp.gamma};
    join_topk();
    launch_planes("predict_score", &s, 1, l2 ? tc::SIDE_NORMS : tc::SIDE_NONE, -1, -1);
    KGE_CUDA(cudaGetLastError());
    return filtered;
}

size_t Engine::debug_fetch(const std::string& what, size_t shard, float* out, size_t capacity) {
    KGE_CUDA(cudaSetDevice((int)cfg_.device_ordinal));
    if (shard >= n_local_) fail(KGE_INVALID_ARGUMENT, "kge_debug_fetch: shard out of range");
    const ShardBuffers& b = shards_[shard];
    const size_t B = cfg_.batch_size, T = cfg_.n_tail(), R = cfg_.n_remote(), D = cfg_.d;
    const float* src = nullptr;
    size_t count = 0;
    if (what == "hidden") { src = b.hid_h; count = R * D; }
    else if (what == "hidden_tail") { src = b.hid_t; count = R * D; }
    else if (what == "tails") { src = b.tails; count = T * D; }
    else if (what == "pred") { src = b.pred; count = B * D; }
    else if (what == "raw_score") { src = b.raw; count = B * T; }
    else if (what == "coeff") { src = b.coeff; count = B * T; }
    else if (what == "d_pred") { src = b.d_pred; count = B * D; }
    else if (what == "d_hidden") { src = b.d_hid_h; count = R * D; }
    else if (what == "grad_recv") { src = b.grad_recv; count = T * D; }
    else if (what == "dense_grad") {
        if (cfg_.world > 1) fail(KGE_INVALID_ARGUMENT, "kge_debug_fetch: 'dense_grad' is spread over the processes; fetch it with one process");
        if (fuse_dense_ && n_dense_ <= capacity) restore_dense_partial((unsigned)shard);
        src = b.dense_partial; count = n_dense_;
    }
    else if (what == "loss_last") { src = d_loss_last_ + shard; count = 1; }
    else if (what == "exchange_trace") {
        // microseconds since the earliest stamp, [kTraceSlots][XCHG_KINDS][published | wait began | wait ended]; 0 = no stamp
        const size_t n = (size_t)kTraceSlots * XCHG_KINDS * 3;
        if (!d_xchg_trace_) fail(KGE_INVALID_ARGUMENT, "kge_debug_fetch: exchange_trace needs KGE_EXCHANGE_TRACE=1 in the environment");
        if (n > capacity) fail(KGE_INVALID_ARGUMENT, msg() << "kge_debug_fetch: 'exchange_trace' needs room for " << n << " floats");
        KGE_CUDA(cudaStreamSynchronize(stream_));
        std::vector<unsigned long long> stamps(n);
        KGE_CUDA(cudaMemcpy(stamps.data(), d_xchg_trace_, n * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
        unsigned long long base = ~0ull;
        for (unsigned long long v : stamps) if (v && v < base) base = v;
        for (size_t i = 0; i < n; ++i) out[i] = stamps[i] ? (float)((double)(stamps[i] - base) * 1e-3) + 1e-3f : 0.f;
        return n;
    }
    else fail(KGE_INVALID_ARGUMENT, msg() << "kge_debug_fetch: unknown buffer '" << what << "'");
    if (count > capacity) fail(KGE_INVALID_ARGUMENT, msg() << "kge_debug_fetch: '" << what << "' needs room for " << count << " floats");
    KGE_CUDA(cudaStreamSynchronize(stream_));
    if (count && (src == b.raw || src == b.coeff)) KGE_CUDA(cudaMemcpy2D(out, T * 4, src, score_ld_ * 4, T * 4, B, cudaMemcpyDeviceToHost));
    else if (count) KGE_CUDA(cudaMemcpy(out, src, count * 4, cudaMemcpyDeviceToHost));
    return count;
}

}  // namespace kge
