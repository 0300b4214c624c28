// Stand-in for the one third-party header that torch's functorch headers name but torch does not ship.  They use it
// only in inline (de)serialisation helpers of interpreter metadata, which nothing here calls: declarations are enough.
#pragma once

#include <string>

namespace nlohmann {

class json {
 public:
  json();
  template <typename T> json(const T&);
  template <typename T> json& operator=(const T&);
  template <typename K> json& operator[](const K&);
  template <typename K> const json& operator[](const K&) const;
  template <typename K> const json& at(const K&) const;
  template <typename T> T get() const;
  template <typename T> void get_to(T&) const;
  template <typename T> operator T() const;
  static json parse(const std::string&);
  std::string dump() const;
};

}  // namespace nlohmann
