// Tables that several owners share.
#pragma once

#include <map>
#include <memory>
#include <mutex>

namespace vqb {

// One table a key, formed by the first that asks for it and held for as long
// as any of its owners holds it. Who asks for a key that is being formed
// waits for it; other keys are formed meanwhile.
template <class Key, class T>
class SharedTables {
  public:
    template <class Make>
    std::shared_ptr<const T> get(const Key &key, Make &&make) {
        std::shared_ptr<Entry> entry;
        {
            std::lock_guard<std::mutex> lock(mu_);
            std::shared_ptr<Entry> &at = entries_[key];
            if (!at) at = std::make_shared<Entry>();
            entry = at;
        }
        std::lock_guard<std::mutex> lock(entry->mu);
        std::shared_ptr<const T> table = entry->table.lock();
        if (!table) entry->table = table = make();
        return table;
    }

  private:
    struct Entry {
        std::mutex mu;
        std::weak_ptr<const T> table;
    };
    std::mutex mu_;
    std::map<Key, std::shared_ptr<Entry>> entries_;
};

}  // namespace vqb
